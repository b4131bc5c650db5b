// Block-scaled FP8 GEMM for few activation rows per weight matrix (dense decode, experts with some rows each).
//
//   C[m,n] = out_t( sum_kb a_s[m,kb] * b_s[n/128,kb] * sum_{k in kb} A[m,k] * B[n,k] )      (as in gemm.cu)
//
// gemm.cu puts 128 activation rows on the lanes of the accumulator; with 1 to 64 rows most of what it stages, multiplies
// and promotes is padding, and its tiles are wide, so a weight matrix makes few of them.  Here the operands trade
// places: 128 WEIGHT rows are the M side of the tcgen05.mma, the activation rows are its N side, which comes in steps
// of 16.  A tile of the accumulator is 128 weight rows (lanes) x up to NT activation rows (columns), and the work per
// tile (staged bytes, MMA, promotion) follows the rows it has, rounded up to 16, chosen per tile at run time.
//
// What bounds it: HBM, as the weights are read once and everything else is small.  So the design is about bytes in
// flight and about having none of the SMs wait: two CTAs per SM (NT <= 64) with about 100 KB of ring each, the
// producer running ahead over tile boundaries, and K split over the CTAs of a thread-block cluster where a matrix has
// fewer tiles than the GPU has CTA slots; the cluster adds its partial sums through distributed shared memory in
// ascending K order, without a second kernel.  Launched after the quantizer with programmatic serialization, the
// producer fetches its first weight tiles while the quantizer still runs.
//
// Roles (one CTA): warp 0 issues the TMA loads (all lanes: one box of 16 rows, or one gather of 4 rows, per lane and
// slab), warp 1 issues the MMAs, warp 2 prepares the scales (a_s * b_s of eight slabs at a time, one product per
// column, in shared memory), warps 4.. promote: TMEM -> registers, acc += partial * scale, then store.  Next to HBM the
// shared-memory port is the limit: 64 rows stage 24 KB a slab and the MMA reads them back, 384 clocks at 128 bytes a
// clock; see the promotion for what the scales add.
// Every mbarrier wait is bounded as in gemm.cu (status word, no trap).
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "gemm_rows.cuh"

namespace sglb200 {

template <int NT_, int kPromoWarps_, int kStages_, int kAccBufs_, int kCtasPerSm_>
struct RowsCfg {
  static constexpr int NT = NT_, kPromoWarps = kPromoWarps_, kStages = kStages_, kAccBufs = kAccBufs_,
                       kCtasPerSm = kCtasPerSm_;
  static constexpr int kThreads = 128 + kPromoWarps * 32;
  static constexpr int kCW = NT < 32 ? NT : 32;           // columns that a promotion warp takes out of TMEM at once
  static constexpr int kChunks = NT / kCW;
  static constexpr uint32_t kStageBytes = kWBytes + NT * kRowsBK;
  static constexpr int kTmemCols = kAccBufs * NT;
  static_assert((kTmemCols & (kTmemCols - 1)) == 0 && kTmemCols >= 32 && kTmemCols * kCtasPerSm <= 512, "TMEM columns");
  static_assert(NT % 16 == 0 && kStageBytes % 1024 == 0 && kPromoWarps == 4, "tile layout");
};
using Rows16 = RowsCfg<16, 4, 6, 8, 2>;
using Rows32 = RowsCfg<32, 4, 5, 8, 2>;
using Rows64 = RowsCfg<64, 4, 4, 4, 2>;

constexpr int kTileSlots = 4;

template <class Cfg>
struct RowsCtl {
  uint64_t full[Cfg::kStages], empty[Cfg::kStages];
  uint64_t tmem_full[Cfg::kAccBufs], tmem_empty[Cfg::kAccBufs];
  uint64_t sc_full[2], sc_empty[2];
  uint64_t tile_full[kTileSlots], tile_empty[kTileSlots];  // the tiles that the producer took, for the other roles
  RowsTile tile[kTileSlots];                               // n_eff = 0: there is none left
  uint32_t tmem_base;
  int abort_flag;
  int warp_sum[32];
  alignas(16) float sc[2][kScBatch][Cfg::NT];  // a_s * b_s per slab and column (columns in the order of frag_column)
  // (grouped: followed by tiles_before[experts + 1], the token tiles of the experts before e)
};

__device__ int g_rows_status = 0;  // 0 ok, 1 = a pipeline wait expired

// kCounter (grouped): there may be more tiles than CTAs, see take_tile.
template <class Cfg, bool kGrouped, bool kCounter>
__global__ void __launch_bounds__(Cfg::kThreads, Cfg::kCtasPerSm)
    fp8_rows_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                         const RowsParams p) {
  constexpr int NT = Cfg::NT, kStages = Cfg::kStages, kAccBufs = Cfg::kAccBufs, kCW = Cfg::kCW, kChunks = Cfg::kChunks;
  constexpr bool kPush = !kGrouped && NT == 64;  // how a cluster exchanges its partial sums
  static_assert(NT * kPartPitch <= kStages * Cfg::kStageBytes / 4 &&
                    (NT / 2 + kMaxSplits - 1) * kPartPair <= kStages * Cfg::kStageBytes / 4,
                "the partial sums fit the ring");
  constexpr uint32_t kStageBytes = Cfg::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  RowsCtl<Cfg>* ctl = reinterpret_cast<RowsCtl<Cfg>*>(tiles + kStages * kStageBytes);
  int* tiles_before = reinterpret_cast<int*>(ctl + 1);  // grouped: token tiles before every expert
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &ctl->abort_flag;

  ptx::launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&ctl->full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->empty[s]), 1);
    }
    for (int b = 0; b < kAccBufs; ++b) {
      ptx::mbar_init(ptx::smem_u32(&ctl->tmem_full[b]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->tmem_empty[b]), Cfg::kPromoWarps);
    }
    for (int d = 0; d < 2; ++d) {
      ptx::mbar_init(ptx::smem_u32(&ctl->sc_full[d]), 32);
      ptx::mbar_init(ptx::smem_u32(&ctl->sc_empty[d]), Cfg::kPromoWarps);
    }
    for (int d = 0; kCounter && d < kTileSlots; ++d) {
      ptx::mbar_init(ptx::smem_u32(&ctl->tile_full[d]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->tile_empty[d]), Cfg::kPromoWarps + 2);
    }
    ctl->abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&map_w);
    ptx::tma_prefetch_desc(&map_a);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  if constexpr (kGrouped) {
    ptx::grid_dependency_wait();
    rows_count_tiles<NT, Cfg::kThreads>(p, tiles_before, ctl->warp_sum);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  const int splits = p.splits;
  const int rank = splits > 1 ? (int)(blockIdx.x % splits) : 0;
  const int tile_first = splits > 1 ? (int)(blockIdx.x / splits) : (int)blockIdx.x;
  const int tile_step = splits > 1 ? (int)(gridDim.x / splits) : (int)gridDim.x;
  const int num_tiles = (kGrouped ? tiles_before[p.num_experts] : p.tiles_m) * p.tiles_n;
  const int kb_begin = rank * p.kb_total / splits, kb_stop = (rank + 1) * p.kb_total / splits;

  // The tiles of this CTA, one call after the other.  With kCounter the producer takes them, from a counter that the CTAs
  // share, and hands them to the other roles through a ring; otherwise they are dealt out in turn and every role counts for
  // itself.  `t` and `x` are the caller's; false = none left, or a wait expired.
  // The counter is for experts with more tiles than CTAs: those that HBM serves faster then take more of them, and a last
  // round that is part full spreads over all SMs.  Dealt out in turn, the CTAs of 256 experts of 7168 x 2048 with 64 tokens
  // ended between 849 and 940 us of the first product; the layer took 1 419 us and takes 1 369; 128 experts of 2048 x 768
  // from a graph, 32 tokens 117.5 and 108.7, 16 tokens 86.3 and 84.2.  Where a CTA has a tile or none the ring only costs (one
  // token, 8 experts of 4096 x 1408 30.0 us, in turn 29.1; 16 experts of 2048 x 768 23.0 and 22.6), so the host leaves it out
  // where the number of rows bounds the tiles.  Both ways in one kernel, chosen by the tiles there are, 31.1 and 23.7: its
  // code is fetched anew in every launch.  Weights of the first tile asked for before its row ids, so that these wait behind
  // them, cost another 1 to 2 us.
  const uint32_t bar_tile_full0 = ptx::smem_u32(&ctl->tile_full[0]), bar_tile_empty0 = ptx::smem_u32(&ctl->tile_empty[0]);
  uint32_t ts = 0, tph = 0;
  auto take_tile = [&](int& t, RowsTile& x, bool first, bool one_thread) -> bool {
    if constexpr (kCounter) {
      if (!ROWS_WAIT(bar_tile_full0 + ts * 8, tph)) {
        *abort_flag = 1;
        return false;
      }
      x = ctl->tile[ts];
      if (!one_thread) __syncwarp();  // (every lane has read it)
      if (one_thread || lane == 0) ptx::mbar_arrive(bar_tile_empty0 + ts * 8);
      if (++ts == (uint32_t)kTileSlots) ts = 0, tph ^= 1u;
      return x.n_eff > 0;
    } else {
      t = first ? tile_first : t + tile_step;
      if (t >= num_tiles) return false;
      x = rows_tile<NT, kGrouped>(p, tiles_before, t);
      return true;
    }
  };

  if (warp == 0) {
    // ------------------------------ TMA producer (all lanes) ------------------------------
    const uint32_t bar_empty0 = ptx::smem_u32(&ctl->empty[0]), bar_full0 = ptx::smem_u32(&ctl->full[0]);
    const uint32_t tiles0 = ptx::smem_u32(tiles);
    // Slabs whose weights are already on their way: the first tile's, fetched before the activations can be.
    int ahead = 0;
    if (!kGrouped) {
      if (p.early_weights && tile_first < num_tiles) {
        const RowsTile x = rows_tile<NT, kGrouped>(p, tiles_before, tile_first);
        ahead = min(kStages, kb_stop - kb_begin);
        if (lane == 0)
          for (int s = 0; s < ahead; ++s) {
            ptx::mbar_arrive_expect_tx(bar_full0 + s * 8, kWBytes + x.n_eff * kRowsBK);
            ptx::tma_load_3d(tiles0 + s * kStageBytes, &map_w, bar_full0 + s * 8, (kb_begin + s) * kRowsBK, x.n_tile * kRowsBM, 0);
          }
        __syncwarp();
      }
      ptx::grid_dependency_wait();
    }
    uint32_t s = 0, ph = 0;
    bool alive = true;
    auto publish = [&](const RowsTile& x) -> bool {
      if (!ROWS_WAIT(bar_tile_empty0 + ts * 8, tph ^ 1u)) {
        *abort_flag = 1;
        return false;
      }
      if (lane == 0) {
        ctl->tile[ts] = x;
        ptx::mbar_arrive(bar_tile_full0 + ts * 8);
      }
      if (++ts == (uint32_t)kTileSlots) ts = 0, tph ^= 1u;
      return true;
    };
    int t_next = 0;
    for (int t = tile_first; t < num_tiles && alive; t = kCounter ? __shfl_sync(0xffffffffu, t_next, 0) : t + tile_step) {
      const RowsTile x = rows_tile<NT, kGrouped>(p, tiles_before, t);
      if (kCounter && !publish(x)) break;
      const bool gather = kGrouped && p.gather_topk > 0;
      int r[4] = {0, 0, 0, 0};
      if (gather && lane * 4 < x.n_eff) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int id = p.sorted_ids[x.row0 + lane * 4 + j];
          r[j] = id < p.numel ? id / p.gather_topk : 0;  // (padding fetches a valid row; its scale is zero)
        }
      }
      const uint32_t bytes = kWBytes + x.n_eff * kRowsBK;
      for (int kb = kb_begin; kb < kb_stop; ++kb) {
        const uint32_t bar = bar_full0 + s * 8, dst = tiles0 + s * kStageBytes;
        const int k0 = kb * kRowsBK;
        // (late enough that the next tile is taken by a CTA that can start it, early enough that the answer is not waited for)
        if (kCounter && lane == 0 && kb == max(kb_begin, kb_stop - kStages))
          t_next = num_tiles > (int)gridDim.x ? atomicAdd(p.next_tile, 1) + (int)gridDim.x : num_tiles;
        if (ahead > 0) {
          --ahead;
        } else {
          if (!ROWS_WAIT(bar_empty0 + s * 8, ph ^ 1u)) { *abort_flag = 1; alive = false; break; }
          if (lane == 0) {
            ptx::mbar_arrive_expect_tx(bar, bytes);
            ptx::tma_load_3d(dst, &map_w, bar, k0, x.n_tile * kRowsBM, x.expert);
          }
          __syncwarp();
        }
        if (gather) {
          if (lane * 4 < x.n_eff) ptx::tma_gather4(dst + kWBytes + lane * (4 * kRowsBK), &map_a, bar, k0, r[0], r[1], r[2], r[3]);
        } else if (lane * 16 < x.n_eff) {
          ptx::tma_load_2d(dst + kWBytes + lane * (16 * kRowsBK), &map_a, bar, k0, x.row0 + lane * 16);
        }
        if (++s == (uint32_t)kStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    if (kCounter && alive) publish(RowsTile{0, 0, 0, 0});
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (ptx::elect_one()) {
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // see gemm.cu
      const uint32_t desc_lo0 = ((ptx::smem_u32(tiles) & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t bar_full0 = ptx::smem_u32(&ctl->full[0]), bar_empty0 = ptx::smem_u32(&ctl->empty[0]);
      const uint32_t bar_tfull0 = ptx::smem_u32(&ctl->tmem_full[0]), bar_tempty0 = ptx::smem_u32(&ctl->tmem_empty[0]);
      uint32_t s = 0, ph = 0, buf = 0, aph = 0;
      bool alive = true;
      int t = 0;
      RowsTile x;
      for (bool first = true; alive && take_tile(t, x, first, true); first = false) {
        const uint32_t idesc = ptx::make_idesc_e4m3_f32(kRowsBM, x.n_eff);
        for (int kb = kb_begin; kb < kb_stop; ++kb) {
          if (!ROWS_WAIT(bar_tempty0 + buf * 8, aph ^ 1u) || !ROWS_WAIT(bar_full0 + s * 8, ph)) {
            *abort_flag = 1;
            alive = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t a_lo = desc_lo0 + s * (kStageBytes >> 4), b_lo = a_lo + (kWBytes >> 4);
#pragma unroll
          for (int k = 0; k < kRowsBK / 32; ++k)
            ptx::mma_f8f6f4(tmem_base + buf * NT, ptx::pack_f32x2(a_lo + 2 * k, kDescHi), ptx::pack_f32x2(b_lo + 2 * k, kDescHi),
                            idesc, k > 0 ? 1u : 0u);
          ptx::mma_commit(bar_empty0 + s * 8);
          ptx::mma_commit(bar_tfull0 + buf * 8);
          if (++s == (uint32_t)kStages) {
            s = 0;
            ph ^= 1u;
          }
          if (++buf == (uint32_t)kAccBufs) {
            buf = 0;
            aph ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------ scales ------------------------------
    // Lane l prepares columns l, l + 32, ..: eight slabs per step, all loads of a step in flight together and one
    // step ahead of the promotion (two slots).
    constexpr int kPer = (NT + 31) / 32;
    const uint32_t bar_full0 = ptx::smem_u32(&ctl->sc_full[0]), bar_empty0 = ptx::smem_u32(&ctl->sc_empty[0]);
    ptx::grid_dependency_wait();
    uint32_t d = 0, dph = 0;
    bool alive = true;
    int t = 0;
    RowsTile x;
    for (bool first = true; alive && take_tile(t, x, first, false); first = false) {
      const float* b_row = p.b_s + ((int64_t)x.expert * p.nb_total + x.n_tile) * p.kb_total;
      const float* a_row[kPer];
      bool on[kPer];
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int j = lane + 32 * i;
        on[i] = j < x.n_eff;
        int64_t row = x.row0 + j;
        if (kGrouped) {
          if (on[i] && p.gather_topk > 0) {
            const int id = p.sorted_ids[row];
            on[i] = id < p.numel;
            row = on[i] ? id / p.gather_topk : 0;
          }
        } else {
          on[i] = row < p.M;
        }
        a_row[i] = p.a_s + row * p.as_stride_m;
      }
      for (int kb0 = kb_begin; kb0 < kb_stop; kb0 += kScBatch) {
        float v[kPer][kScBatch];
#pragma unroll
        for (int b = 0; b < kScBatch; ++b) {
          const float bs = kb0 + b < kb_stop ? __ldg(b_row + kb0 + b) : 0.f;
#pragma unroll
          for (int i = 0; i < kPer; ++i)
            v[i][b] = on[i] && kb0 + b < kb_stop ? __ldg(a_row[i] + (int64_t)(kb0 + b) * p.as_stride_k) * bs : 0.f;
        }
        if (!ROWS_WAIT(bar_empty0 + d * 8, dph ^ 1u)) { *abort_flag = 1; alive = false; break; }
#pragma unroll
        for (int b = 0; b < kScBatch; ++b)
#pragma unroll
          for (int i = 0; i < kPer; ++i)
            if (lane + 32 * i < NT) ctl->sc[d][b][frag_column(lane + 32 * i)] = v[i][b];
        ptx::mbar_arrive(bar_full0 + d * 8);
        d ^= 1u;
        if (d == 0) dph ^= 1u;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------ promotion + store ------------------------------
    // The accumulator is read as fragments of 16 lanes x 8 columns: a thread holds four of the warp's 32 weight rows
    // (lane / 4 + 8 i) in two neighbouring columns (2 (lane % 4), + 1) of every eight, so that a scale it reads serves four
    // values.  With a lane per weight row every lane needs every column's scale, and a shared-memory read delivers 128
    // bytes a clock however many lanes ask for the same word: 256 clocks a slab for 64 rows beside 384 of operands, 64 this
    // way.  64 rows by 36864 x 7168, with the quantizer: 52.2 us with a lane per weight row, 49.7 so; 4096 x 4096 11.5
    // and 11.3.
    const int q = warp & 3;
    const uint32_t bar_tfull0 = ptx::smem_u32(&ctl->tmem_full[0]), bar_tempty0 = ptx::smem_u32(&ctl->tmem_empty[0]);
    const uint32_t bar_sfull0 = ptx::smem_u32(&ctl->sc_full[0]), bar_sempty0 = ptx::smem_u32(&ctl->sc_empty[0]);
    const uint32_t taddr0 = tmem_base + ((uint32_t)(q * 32) << 16);
    const uint32_t sc0 = ptx::smem_u32(&ctl->sc[0][0][0]) + (lane & 3) * 16;
    constexpr int kBlocks = kCW / 16, kRegs = 8 * kBlocks;  // 16-column blocks of a chunk; values of half a chunk (16 lanes)
    ptx::grid_dependency_wait();
    uint32_t buf = 0, aph = 0, d = 0, dph = 0;
    bool alive = true, arrived = false, waited = false;
    int t = 0;
    RowsTile x;
    for (bool first = true; alive && take_tile(t, x, first, false); first = false) {
      const int active = (x.n_eff + kCW - 1) / kCW;  // chunks that hold columns of the tile
      float acc[kChunks][2][kRegs];                  // chunk, 16-lane half, [block][8 columns of it][row lane / 4, + 8][2]
#pragma unroll
      for (int i = 0; i < kChunks; ++i)
#pragma unroll
        for (int j = 0; j < kRegs; ++j) acc[i][0][j] = acc[i][1][j] = 0.f;
      const int slabs = kb_stop - kb_begin;
      for (int g = 0; g < slabs; ++g) {
        const int b = g & (kScBatch - 1);
        if ((b == 0 && !ROWS_WAIT(bar_sfull0 + d * 8, dph)) || !ROWS_WAIT(bar_tfull0 + buf * 8, aph)) {
          *abort_flag = 1;
          alive = false;
          break;
        }
        ptx::tc_fence_after();
        if (kPush && splits > 1 && g == slabs - 1) {  // the operands have been consumed: the ring may be written
          ptx::cluster_arrive();
          arrived = true;
        }
        const uint32_t taddr = taddr0 + buf * NT, sc = sc0 + (d * kScBatch + b) * (NT * 4);
#pragma unroll
        for (int i = 0; i < kChunks; ++i) {
          if (i < active) {
            uint32_t r[2][kRegs];
            float4 s4[kBlocks];
            ptx::tmem_ld_16x256<2 * kBlocks>(taddr + i * kCW, r[0]);
            ptx::tmem_ld_16x256<2 * kBlocks>(taddr + i * kCW + (16u << 16), r[1]);
#pragma unroll
            for (int w = 0; w < kBlocks; ++w) s4[w] = ptx::lds_f32x4(sc + (i * kBlocks + w) * 64);
            ptx::tmem_ld_wait();
            if (i == active - 1) {
              ptx::tc_fence_before();
              ptx::mbar_arrive_if(bar_tempty0 + buf * 8, lane == 0);
            }
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
              for (int w = 0; w < kBlocks; ++w) {
                float* a = acc[i][hf] + 8 * w;
                const uint32_t* v = r[hf] + 8 * w;
                ptx::fma2(a[0], a[1], v[0], v[1], s4[w].x, s4[w].y);
                ptx::fma2(a[2], a[3], v[2], v[3], s4[w].x, s4[w].y);
                ptx::fma2(a[4], a[5], v[4], v[5], s4[w].z, s4[w].w);
                ptx::fma2(a[6], a[7], v[6], v[7], s4[w].z, s4[w].w);
              }
          }
        }
        if (b == kScBatch - 1 || g == slabs - 1) {
          __syncwarp();
          ptx::mbar_arrive_if(bar_sempty0 + d * 8, lane == 0);
          d ^= 1u;
          if (d == 0) dph ^= 1u;
        }
        if (++buf == (uint32_t)kAccBufs) {
          buf = 0;
          aph ^= 1u;
        }
      }
      if (!alive) break;
      if (kPush && splits > 1) {
        ptx::cluster_wait();
        waited = true;
#pragma unroll
        for (int i = 0; i < kChunks; ++i)
          if (i < active) rows_cluster_put<2 * kBlocks>(p, x, rank, ptx::smem_u32(tiles), acc[i][0], acc[i][1], i * kCW, q, lane);
        continue;
      }
      if (!kPush && splits > 1) {
        // this CTA's partial sums, [column][weight row], over its ring: every slab has been consumed, and a cluster
        // works on one tile only
        float* part = reinterpret_cast<float*>(tiles) + 2 * (lane & 3) * kPartPitch + q * 32 + (lane >> 2);
#pragma unroll
        for (int i = 0; i < kChunks; ++i)
          if (i < active) {
#pragma unroll
            for (int j = 0; j < kRegs; ++j) {
              float* at = part + (i * kCW + (j >> 2) * 8 + (j & 1)) * kPartPitch + ((j >> 1) & 1) * 8;
              at[0] = acc[i][0][j];
              at[16] = acc[i][1][j];
            }
          }
        continue;
      }
      // Eight columns (output rows) at a time: rounded and transposed in registers, so that a lane has eight neighbouring
      // values of one output row and four lanes write 64 contiguous bytes.
      const int n0 = x.n_tile * kRowsBM + q * 32;
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (!kGrouped && p.bias != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = min(n0 + 8 * i + (lane >> 2), (int)p.N - 1);
          bias[i] = p.out_fp16 ? __half2float(static_cast<const __half*>(p.bias)[n])
                               : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[n]);
        }
      }
      const int n = n0 + (lane & 3) * 8;  // first of the eight values this lane writes (N is a multiple of 8)
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
#pragma unroll
        for (int w = 0; w < kBlocks; ++w) {
          const int col0 = i * kCW + w * 16;
          if (col0 < x.n_eff) {
            // destination row and routing weight of column col0 + lane % 16; -1 = not stored
            int dst = x.row0 + col0 + (lane & 15);
            float wt = 1.f;
            if (kGrouped) {
              if (p.scatter) {
                const int id = p.sorted_ids[dst];
                dst = id < p.numel ? id : -1;
                if (p.row_weights != nullptr && dst >= 0) wt = __ldg(p.row_weights + id);
              }
            } else if (dst >= p.M) {
              dst = -1;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int c = 8 * u + 2 * (lane & 3);
              const float w0 = kGrouped ? __shfl_sync(0xffffffffu, wt, c) : 1.f;
              const float w1 = kGrouped ? __shfl_sync(0xffffffffu, wt, c + 1) : 1.f;
              uint32_t m[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {  // weight rows lane / 4 + 8 k
                const float* a = acc[i][k >> 1] + 8 * w + 4 * u + 2 * (k & 1);
                float v0 = a[0], v1 = a[1];
                if (kGrouped) v0 *= w0, v1 *= w1;
                else v0 += bias[k], v1 += bias[k];
                if (p.out_fp16) {
                  const __half2 o = __floats2half2_rn(v0, v1);
                  m[k] = *reinterpret_cast<const uint32_t*>(&o);
                } else {
                  const __nv_bfloat162 o = __floats2bfloat162_rn(v0, v1);
                  m[k] = *reinterpret_cast<const uint32_t*>(&o);
                }
              }
              const int row = __shfl_sync(0xffffffffu, dst, 8 * u + (lane >> 2));
              const uint4 v = ptx::transpose_frags(m, lane);
              if (row >= 0 && n < p.N) *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.C) + (int64_t)row * p.N + n) = v;
            }
          }
        }
      }
    }
    if (kPush && splits > 1 && !waited) {  // (a wait expired: the others must not wait for this warp)
      if (!arrived) ptx::cluster_arrive();
      ptx::cluster_wait();
    }
  }

  // ------------------------------ sum over the CTAs of a cluster ------------------------------
  if (kPush && splits > 1) {
    __syncwarp();
    if (warp < 4) {
      ptx::cluster_arrive();
      ptx::cluster_wait();
    }
    ptx::cluster_arrive();
    ptx::cluster_wait();  // (nothing crosses the cluster after this: a CTA may leave)
    const RowsTile x = rows_tile<NT, kGrouped>(p, tiles_before, tile_first);
    if (ctl->abort_flag == 0) rows_cluster_get(p, x, rank, ptx::smem_u32(tiles), warp, Cfg::kThreads / 32, lane);
  } else if (!kGrouped && splits > 1) {
    __syncwarp();
    ptx::cluster_sync();
    const RowsTile x = rows_tile<NT, kGrouped>(p, tiles_before, tile_first);
    if (ctl->abort_flag == 0) {
      if (splits <= 8) rows_cluster_sum<8>(p, x, rank, ptx::smem_u32(tiles), tid, Cfg::kThreads);
      else rows_cluster_sum<kMaxSplits>(p, x, rank, ptx::smem_u32(tiles), tid, Cfg::kThreads);
    }
    ptx::cluster_sync();  // no CTA leaves while another reads its shared memory
  }

  // ------------------------------ teardown ------------------------------
  ptx::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag != 0 && tid == 0) {
    atomicExch(&g_rows_status, 1);
    // give TMA copies that may still be in flight time to land before the CTA's shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

template <class Cfg, bool kGrouped>
static size_t rows_smem_bytes(int num_experts) {
  return (size_t)Cfg::kStages * Cfg::kStageBytes + sizeof(RowsCtl<Cfg>) + 1024 + (kGrouped ? sizeof(int) * (num_experts + 1) : 0);
}

// `pdl`: the launch may overlap the end of the kernel before it in the stream (the kernel waits by itself).
template <class Cfg, bool kGrouped, bool kCounter>
static int launch_rows(const CUtensorMap& mw, const CUtensorMap& ma, const RowsParams& p, int64_t max_tiles, bool pdl,
                       cudaStream_t st) {
  auto kern = fp8_rows_gemm_kernel<Cfg, kGrouped, kCounter>;
  const size_t smem = rows_smem_bytes<Cfg, kGrouped>(p.num_experts);
  static thread_local bool attr_set[64] = {false};  // the opt-in is per function and per device
  int dev = 0;
  SGLB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)rows_smem_bytes<Cfg, kGrouped>(kMaxExperts)));
    if (!kGrouped) SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  const int64_t slots = (int64_t)sm_count() * Cfg::kCtasPerSm;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.splits > 1 ? max_tiles * p.splits : (max_tiles < slots ? max_tiles : slots)), 1, 1);
  cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = 0;
  if (p.splits > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)p.splits;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (pdl) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  SGLB_CUDA(cudaLaunchKernelEx(&cfg, kern, mw, ma, p));
  return SGLB200_OK;
}

// Never launched: the occupancy questions below are asked about it.
__global__ void cluster_probe_kernel() {}

const ClusterFits& cluster_fits() {
  constexpr int kAlone = 120 * 1024, kPaired = 104 * 1024;  // of 227 KB: one and two CTAs per SM
  const auto ask = [](int s, int per_sm) -> int64_t {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)s, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s, 1, 1), cfg.blockDim = dim3(256, 1, 1);
    cfg.dynamicSmemBytes = per_sm == 1 ? kAlone : kPaired;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(cluster_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlone) != cudaSuccess ||
        cudaFuncSetAttribute(cluster_probe_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, cluster_probe_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  };
  static std::once_flag once[64];
  static ClusterFits known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    static const ClusterFits portable = cluster_fits_of([](int, int) -> int64_t { return 0; }, 148);
    return portable;
  }
  std::call_once(once[dev], [&] { known[dev] = cluster_fits_of(ask, sm_count()); });
  return known[dev];
}

template <class Cfg>
static int rows_dense_cfg(const void* A, const void* B, RowsParams& p, int64_t K, bool pdl, cudaStream_t st) {
  CUtensorMap mw, ma;
  int rc = get_tensor_map(B, (uint64_t)K, (uint64_t)p.N, 1, kRowsBM, 3, &mw);
  if (rc) return rc;
  rc = get_tensor_map(A, (uint64_t)K, (uint64_t)p.M, 1, 16, 2, &ma);
  if (rc) return rc;
  p.tiles_m = (int)((p.M + Cfg::NT - 1) / Cfg::NT);
  p.group_m = choose_group_m(p.M, K, Cfg::NT);
  const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n;
  static_assert(Cfg::kCtasPerSm == 2, "rows_splits counts on two");
  p.splits = rows_splits(tiles, p.kb_total, p.M, cluster_fits());
  return launch_rows<Cfg, false, false>(mw, ma, p, tiles, pdl, st);
}

int rows_dense_mm(const void* A, const void* B, const float* a_s, const float* b_s, void* C, const void* bias, int64_t M,
                  int64_t N, int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype, bool after_quantizer,
                  cudaStream_t st) {
  RowsParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = C, p.bias = bias;
  p.M = M, p.N = N, p.as_stride_m = as_stride_m, p.as_stride_k = as_stride_k;
  p.kb_total = (int)((K + kRowsBK - 1) / kRowsBK), p.nb_total = (int)((N + 127) / 128), p.tiles_n = p.nb_total;
  p.out_fp16 = out_dtype;
  p.early_weights = after_quantizer ? 1 : 0;
  p.wait_probes = g_gemm_wait_probes;
  if (M <= 16) return rows_dense_cfg<Rows16>(A, B, p, K, after_quantizer, st);
  if (M <= 32) return rows_dense_cfg<Rows32>(A, B, p, K, after_quantizer, st);
  return rows_dense_cfg<Rows64>(A, B, p, K, after_quantizer, st);
}

// Most token tiles there can be: every expert has at most one partial tile.
static int64_t rows_grouped_tiles(int64_t max_rows, int num_experts, int nt) {
  return std::min(max_rows / nt + num_experts, max_rows / 16);
}
bool rows_grouped_single(int64_t max_rows, int num_experts, int64_t N, int nt) {
  static_assert(Rows32::kCtasPerSm == Rows64::kCtasPerSm, "one number of CTAs for both heights");
  return rows_grouped_tiles(max_rows, num_experts, nt) * ((N + 127) / 128) <= (int64_t)sm_count() * Rows64::kCtasPerSm;
}

template <class Cfg>
static int rows_grouped_cfg(const void* A, int64_t a_rows, const void* B, RowsParams& p, int64_t max_rows, int64_t K, bool pdl,
                            cudaStream_t st) {
  CUtensorMap mw, ma;
  int rc = get_tensor_map(B, (uint64_t)K, (uint64_t)p.N, (uint64_t)p.num_experts, kRowsBM, 3, &mw);
  if (rc) return rc;
  rc = get_tensor_map(A, (uint64_t)K, (uint64_t)a_rows, 1, p.gather_topk > 0 ? 1 : 16, 2, &ma);
  if (rc) return rc;
  p.group_m = choose_group_m(max_rows, K, Cfg::NT);
  p.splits = 1;
  const int64_t tiles = rows_grouped_tiles(max_rows, p.num_experts, Cfg::NT) * p.tiles_n;
  return p.next_tile != nullptr ? launch_rows<Cfg, true, true>(mw, ma, p, tiles, pdl, st)
                                : launch_rows<Cfg, true, false>(mw, ma, p, tiles, pdl, st);
}

int rows_grouped_mm(const void* A, int64_t a_rows, int64_t as_stride, const float* a_s, const void* B, const float* b_s, void* C,
                    const int32_t* cumsum, const int32_t* sorted_ids, const float* row_weights, int64_t max_rows,
                    int64_t numel, int num_experts, int64_t N, int64_t K, int gather_topk, int scatter, int out_dtype, int nt,
                    int32_t* next_tile, bool pdl, cudaStream_t st) {
  RowsParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = C;
  p.M = a_rows, p.N = N, p.as_stride_m = as_stride, p.as_stride_k = 1;
  p.kb_total = (int)((K + kRowsBK - 1) / kRowsBK), p.nb_total = (int)((N + 127) / 128), p.tiles_n = p.nb_total;
  p.out_fp16 = out_dtype, p.num_experts = num_experts, p.cumsum = cumsum, p.sorted_ids = sorted_ids, p.numel = numel;
  p.gather_topk = gather_topk, p.scatter = scatter, p.row_weights = row_weights, p.next_tile = next_tile;
  p.wait_probes = g_gemm_wait_probes;
  switch (nt) {
    case 32: return rows_grouped_cfg<Rows32>(A, a_rows, B, p, max_rows, K, pdl, st);
    case 64: return rows_grouped_cfg<Rows64>(A, a_rows, B, p, max_rows, K, pdl, st);
    default: return fail(SGLB200_E_INVALID, "rows GEMM: %d rows per tile", nt);
  }
}

int rows_gemm_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_rows_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int rows_gemm_status_clear() {
  const int zero = 0;
  SGLB_CUDA(cudaMemcpyToSymbol(g_rows_status, &zero, sizeof(int)));
  return SGLB200_OK;
}

}  // namespace sglb200
