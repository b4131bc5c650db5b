// Block-scaled FP8 GEMM (dense and expert-grouped) for sm_100a.
//
//   C[m,n] = out_t( sum_kb a_s[m,kb] * b_s[n/128,kb] * sum_{k in kb} A[m,k] * B[n,k] )
//
// One persistent CTA per SM walks 128 x BN output tiles: BN = 256 with two TMEM accumulator buffers (the fewest bytes
// per FLOP through shared memory), or BN = 128 with four buffers where one wave of the wide tiles leaves SMs idle.
// Per 128-wide K slab:
//   * warp 0 (one elected lane) issues two TMA tile loads (A 128 rows x 128 B, B BN rows x 128 B,
//     128-byte swizzle) into a shared-memory ring, signalled through `full` mbarriers;
//   * warp 1 (one elected lane) issues four tcgen05.mma kind::f8f6f4 (128 x BN x 32) that write the
//     slab's partial sums into one of the TMEM buffers, then commits the slab to the
//     `empty` barrier of the ring slot and to the `tmem_full` barrier of the buffer;
//   * warps 4-11 (two per TMEM lane quadrant, BN/2 columns each) pull the partial sums out of TMEM with
//     32-column tcgen05.ld, release the buffer, and promote them into float32 register accumulators with the slab's
//     scale a_s[m,kb]*b_s[nb,kb] (DeepSeek-style 128-block float scales cannot be folded into the hardware's
//     power-of-two MX scaling, so promotion runs on the CUDA cores, overlapped with the next slabs' MMAs through the
//     TMEM buffers), two columns per instruction (packed float32 FMA).  Registers are split unevenly (setmaxnreg): 128
//     accumulators per promotion thread leave room for 64 columns in flight;
//   * warp 3 (the scout) runs ahead of the promotion warps: unit coordinates in one of two descriptor slots, the
//     products of activation and weight-block scales, four slabs at a time, in a two-slot ring;
//   * warp 2 (one elected lane) hands finished tiles to the TMA engine: the promotion threads park their rounded
//     part of a tile in shared memory and arrive on an mbarrier, never waiting for each other or for a store.
// What bounds it (M = 4096, N = 36864, K = 7168): the shared-memory port.  A 128 x 256 slab stages 48 KB and the MMAs
// read 48 KB of it, 768 clocks at 128 bytes a clock for 512 clocks of MMA; measured 860 without any promotion and about
// 900 with it.  On the way there, same GPU, back to back (power-limited) in microseconds: 1310 with a 192-wide tile; 1165
// with 256 columns, setmaxnreg and waits that ask before the FMAs and look after them; 1088 with the scales from the
// scout's ring, relaxed hand-backs of tensor memory and the two-step question; 1056 to 1077 (the spread over boxes) with
// the promotion loop unrolled by four, so that buffers, barriers and scales are compile-time (its bookkeeping was a chain
// of dependent instructions as long as the FMAs).  Keeping one TMEM load in flight across the FMAs, chunk by chunk, was
// slower (1250): every extra wait for a load costs more than the overlap gives.  ptxas spills at 168 registers a thread: 4
// to 16 bytes of stores in the dense instances, 60 with experts, 248 where the epilogue activates.
// The epilogue rounds to bf16/fp16, parks the tile in swizzled shared memory, from where TMA stores drain it
// during the next tile; in grouped "scatter" mode it multiplies by the routing weight, parks likewise and writes 128
// contiguous bytes at a time to the token-major row named by sorted_token_ids.
// Scheduling: one wave of 128-wide tiles is taken as it is, or, with few tiles and a long K, split over clusters.  With more, but
// fewer than two waves of 256-wide tiles and a long K, the tiles x slabs space is cut into one equal run of slabs per SM
// (stream-K; a run covers the end of one tile, possibly a whole tile, and the start of the next); otherwise the tiles of a short
// last wave are split along K.  Both write float32 partial sums that a second kernel adds in ascending K order.  In push mode
// (row-parallel layers under tensor parallelism) a tile is stored through the tensor map of the staging buffer of the GPU that
// owns its rows, which folds the reduce-scatter of the all-reduce into the epilogue.
//
// Every mbarrier wait is bounded; on expiry the role raises a flag in shared memory and leaves its loops, the other
// roles sit out their own limits, the CTA sets a status word, drains, frees its TMEM and returns
// (sglb200_gemm_status() reports it).
#include <cuda.h>

#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "common.cuh"
#include "gemm_common.cuh"
#include "ptx_sm100.cuh"
#include "quant_math.cuh"

namespace sglb200 {

constexpr int BM = 128, BK = 128;
constexpr int kScaleBlockN = 128;         // weight scales cover 128 output rows
constexpr int kTmemCols = 512;
constexpr int kEpiWarp0 = 4;              // warp 0 TMA, warp 1 MMA + TMEM owner, warps 4.. promotion + epilogue
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 128 + kEpiWarps * 32;
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kColGroups = kEpiWarps / 4;  // promotion warps per TMEM lane quadrant
constexpr uint32_t kTileBytesA = BM * BK;  // fp8
// A pipeline wait: a bounded run of suspending probes (seconds at most).  `p.wait_probes == kProbesNone` (a
// diagnostic setting) makes every wait give up at once, which exercises the give-up path on a healthy GPU.
// (Measured: also polling the CTA's abort flag between runs of probes, so that one role's expiry ends the others'
// waits early, cost 5 % of the large-M rate; each role sits out its own limit instead.)
// Measurement builds (-DSGLB_TRACE): clock stamps of one promotion warp per column group of CTA 0, per unit.
#ifdef SGLB_TRACE
constexpr int kTraceUnits = 64, kTraceStamps = 8;
__device__ long long g_trace[2][kTraceUnits][kTraceStamps];
#define SGLB_STAMP(i)                                                                                  \
  do {                                                                                                 \
    if (blockIdx.x == 0 && q == 0 && lane == 0 && trace_unit < kTraceUnits) g_trace[cgrp][trace_unit][i] = clock64(); \
  } while (0)
#else
#define SGLB_STAMP(i)
#endif

#define SGLB_WAIT(bar, parity) \
  (p.wait_probes != ptx::kProbesNone && (ptx::mbar_test(bar, parity) || ptx::mbar_wait_quiet(bar, parity)))

// What a launch computes.  kActivated: the gate and up projections of the experts, of which a tile takes 128 columns each
// (columns 0-127 of its accumulators and 128-255), so that the epilogue has both factors of 128 activated values and a whole
// quantisation group of every row, and writes codes and scales instead of 16-bit products that another launch reads back.
// 131072 rows through 128 experts of 2048 x 768 (Zipf routing, sustained, both ways on one GPU): product 493 us + activation 117
// -> 550; 32768 rows, 256 experts of 7168 x 2048: 1 970 + 147 -> 1 979.  The epilogue's exponentials and reciprocals are 2 048
// clocks a tile of the special-function units, which the next tile's first two slabs hide in part.  Four stages of operands,
// for which there is room: 562 and 2 063.
// kOnce: a dense product whose CTAs store at most one tile each, when its last slab has been multiplied (a single wave), or none
// (partial sums only): the staging area then lies in the operand ring, which has room for one stage more.  A slab of a single
// wave takes 1 100 clocks, most of them the way from DRAM and L2 to shared memory (of many waves 850: other rows' CTAs have
// brought the weights), so it is bytes in flight that count.  Us with the quantizer, ring of three stages -> four, both in turn
// on one GPU: 257 x 10240 x 8192 47.6 -> 44.9, 512 x 7168 x 16384 86.3 -> 82.1, 192 x 10240 x 8192 40.8 -> 38.2.
// Shorter K pays with the early weights below, from 12 slabs and 32 CTAs on, 96 where there are more than 128 rows and the CTAs of
// one column ask for the same weights: 128 x 24576 x 1536 14.5 -> 14.1, 128 x 9216 x 2048 11.0 -> 10.6, 128 x 6144 x 2048 10.1 -> 9.9,
// 256 x 7168 x 2048 (112 CTAs) 11.3 -> 11.0, 900 x 2048 x 2048 (128) 11.6 -> 11.3; not 128 x 3072 x 2048 (24) 10.3 -> 10.5, 128 x 4096 x
// 512 7.1 -> 7.3, 160 x 3072 x 1536 (48) 8.7 -> 8.8, 192 x 4096 x 2048 (64) 9.8 -> 10.1, 384 x 3072 x 1536 (72) 9.1 -> 9.5.
// kSplit: a dense product of few 128-wide tiles and a long K, whose slabs are split over the CTAs of a cluster (`tile_splits`); their
// partial sums meet in distributed shared memory (written once, added once) instead of in global memory and a second launch.
// Beside the ring of five stages lies room for what the other CTAs send; sums fetched from the others' memory after a barrier,
// and then a second one before anybody may leave: 0.7 us more.  What is left of the exchange is about 1.6 us (pushing 0.7 to 1.1,
// barrier 0.6 to 1.0, sum 1.0 to 1.4, against 1.1 for a tile that leaves through TMA).  Us of the layer, before (split-K partial
// sums in global memory, or one CTA a tile) and so: 128 x 4096 x 7168 20.6 -> 14.2, 128 x 2112 x 7168 20.8 -> 13.7, 80 x 3072 x
// 4096 14.1 -> 10.5, 256 x 4096 x 7168 21.8 -> 16.5, 128 x 7168 x 16384 36.1 -> 31.5, 1024 x 1024 x 4096 16.2 -> 14.2.
// 256-wide tiles lost up to 4 us on the exchange of twice the sums.
enum class Form { kDense, kGrouped, kActivated, kOnce, kSplit };

// Tile width BN: 256 columns with two TMEM accumulator buffers, or 128 columns with four (more tiles for the same
// problem: where one wave of wide tiles would leave SMs idle).
template <int BN_, Form kForm = Form::kDense>
struct TileCfg {
  static constexpr int BN = BN_;
  static constexpr bool kInRing = kForm == Form::kOnce;  // the staging area
  static constexpr int kStages = (BN_ >= 256 ? 3 : 5) + (kInRing ? 1 : 0);
  // registers per thread after the split: promotion warps / the others.  The block is launched with 168 x 384 threads:
  // 256 * kPromoRegs + 128 * kOtherRegs <= 64512.
  static constexpr int kPromoRegs = BN_ >= 256 ? 224 : 200;
  static constexpr int kOtherRegs = BN_ >= 256 ? 56 : 104;
  static constexpr int kAccBufs = kTmemCols / BN_;   // TMEM accumulator buffers in flight
  static constexpr int kAccStride = BN_;             // TMEM columns between buffers
  static constexpr int kEpiCols = BN_ / kColGroups;  // columns of a buffer owned by one promotion warp
  static constexpr uint32_t kTileBytesB = BN_ * BK;
  static constexpr uint32_t kStageBytes = kTileBytesA + kTileBytesB;
  // output staging for the TMA store: per 64 columns a [128 rows][64 columns] 2-byte tile in the 128-byte swizzle
  static constexpr int kOutGroups = BN_ / 64;
  static constexpr uint32_t kOutGroupBytes = BM * 64 * 2;
  static constexpr uint32_t kOutBytes = kForm == Form::kActivated ? BM * 128
                                        : kForm == Form::kSplit   ? 60 * 1024
                                                                  : kOutGroups * kOutGroupBytes;
  static constexpr uint32_t kOutOffset = kInRing ? 0 : kStages * kStageBytes;  // of the staging area, from the ring
  static constexpr uint32_t kTileArea = kInRing ? kStages * kStageBytes : kOutOffset + kOutBytes;
  static constexpr int kScBlocks = BN_ > kScaleBlockN ? 2 : 1;
  static constexpr int kWeightRows = kForm == Form::kGrouped ? BM : 1;
  static constexpr int kHalfRows = kForm == Form::kActivated ? BM : 1;
  static_assert(kEpiWarps % 4 == 0 && BN_ % kColGroups == 0 && kEpiCols % 32 == 0 && BN_ % 64 == 0 &&
                    kAccBufs * kAccStride <= kTmemCols && BN_ <= 256 && kStageBytes % 1024 == 0,
                "accumulator layout");
};

__device__ int g_gemm_status = 0;  // 0 ok, 1 = a pipeline wait expired

struct GemmParams {
  const float* a_s;
  const float* b_s;
  void* C;
  const void* bias;
  const int32_t* sorted_ids;   // grouped
  const int32_t* expert_ids;   // grouped
  const int32_t* num_rows_dev; // grouped: rows in use (multiple of 128)
  const float* row_weights;    // grouped, optional: of the rows that are scattered, or stored in sorted order with padding to skip
  int64_t M;                   // dense: rows of A; grouped: max rows
  int64_t N, K;
  int64_t as_stride_m, as_stride_k;
  int64_t numel;               // grouped scatter: valid ids are < numel
  int kb_total;                // ceil(K/128)
  int full_units;              // dense: the first `full_units` tiles are one unit each ...
  int splits;                  // ... and every later tile is cut into `splits` units along K (1 = none)
  int kb_per_split;            // K slabs per unit of a split tile
  float* partial;              // float32 partial sums of the split tiles: [slot][column / 4][row][4]
  int nb_total;                // ceil(N/128): weight scale blocks along N
  int tiles_n;                 // ceil(N/BN)
  int scatter;
  int out_fp16;
  int tma_out;                 // rows of C are written with TMA tile stores (map_c is valid)
  int group_m;                 // m-tiles per rasterization group
  // push mode (row-parallel layers): the output rows are owned in equal blocks by `world` GPUs and each tile
  // is stored into its owner's staging buffer [source rank][rows per owner][N] through that buffer's tensor map
  const CUtensorMap* push_maps;  // [world] in global memory, nullptr = ordinary output through map_c
  int push_rows_per_owner;       // a multiple of BM
  int push_rank;                 // this GPU's slot in the owners' staging buffers
  // stream-K mode (fewer than two waves of tiles): the tiles x slabs space is cut into `sk_ctas` equal runs of
  // `sk_share` slabs, one per CTA; a run covers at most `sk_pieces` tiles (the end of one, the start of the next,
  // with a whole tile between them when sk_share exceeds kb_total)
  int sk_share;                  // 0 = off; otherwise <= (sk_pieces - 1) * kb_total
  int sk_ctas;
  int sk_pieces;                 // 2 or 3
  int sk_total;                  // tiles * kb_total
  int early_weights;             // the weights may be read before the predecessor in the stream has finished (kOnce, kSplit)
  uint32_t wait_probes;          // probes after which a pipeline wait gives up
  int skip_padding;              // grouped: nobody reads the rows of a 32-row quadrant that is all padding (sorted_ids >= numel)
  float* act_s;                  // activated form: C holds codes [row][N / 2], this their scales [row][N / 256]
};

// What the scout warp prepares for the promotion warps while they work on the previous unit: where the unit lies, so that
// a promotion warp starts it with a few shared-memory reads instead of integer divisions, and, through a ring of its
// own, the slabs' scales.
struct UnitDesc {
  int m_tile, n_tile, expert, kb_begin;
  int kb_stop, split, slot, live;  // live: leading 32-row quadrants of the tile with rows that count
};
constexpr int kScSlabs = 4;  // slabs per slot of the scale ring: one 16-byte read per promotion thread and weight block

template <class Cfg>
struct SharedCtl {
  alignas(16) float sc[2][Cfg::kScBlocks][BM][kScSlabs];  // a_s * b_s: slot, weight block of the tile, tile row, slab
  UnitDesc desc[2];
  float row_w[2][Cfg::kWeightRows];  // grouped, rows stored in sorted order: their routing weights, a slot as the descriptor's
  uint64_t sc_full[2];     // the slot is written (every scout lane arrives)
  uint64_t sc_empty[2];    // every promotion warp has read it
  uint64_t desc_full[2];   // the descriptor is written (every scout lane arrives)
  uint64_t desc_empty[2];  // every promotion thread has read what it needs from it
  uint64_t full[Cfg::kStages];
  uint64_t empty[Cfg::kStages];
  uint64_t tmem_full[Cfg::kAccBufs];
  uint64_t tmem_empty[Cfg::kAccBufs];
  uint64_t out_full;  // the output staging holds a rounded tile (every promotion thread arrives)
  uint64_t out_free;  // the TMA stores of the previous tile have read the staging (the storing thread arrives)
  // activated form: the two warps of a row quadrant exchange the maxima of their halves of a group
  alignas(16) float2 half_max[2][kColGroups][Cfg::kHalfRows];  // units in turn, column group, row: with NaNs, without
  uint64_t half_full[4];                           // a quadrant's maxima of the unit are written (one lane of each warp)
  uint32_t tmem_base;
  int abort_flag;
};

struct TileCoord {
  int m_tile, n_tile, expert;
};

// Leading 32-row quadrants of a tile that hold rows, by the first ids of the second to the fourth.  An expert's rows come first and
// its padding last, and a tile has a row.
__device__ __forceinline__ int live_quadrants(const GemmParams& p, int id1, int id2, int id3) {
  return 1 + (id1 < p.numel) + (id2 < p.numel) + (id3 < p.numel);
}
__device__ __forceinline__ int live_quadrants(const GemmParams& p, int m_tile) {
  const int32_t* id = p.sorted_ids + (int64_t)m_tile * BM;
  return live_quadrants(p, id[32], id[64], id[96]);
}

// Where a unit lies, and what its tile's rows are: looked up a unit ahead by the roles that must not stall between two tiles.
// The ids stay as they came from memory until the tile is begun, so that nothing waits for them before.
struct TileInfo {
  int m_tile, n_tile, expert, id1, id2, id3;
  __device__ __forceinline__ int live(const GemmParams& p) const { return live_quadrants(p, id1, id2, id3); }
};
template <bool kGrouped>
__device__ __forceinline__ TileInfo tile_info(const GemmParams& p, int tile, int tiles_m, int tiles_n) {
  TileInfo x{0, 0, 0, 0, 0, 0};
  tile_coord(tile, tiles_m, tiles_n, p.group_m, x.m_tile, x.n_tile);
  if (kGrouped) {
    x.expert = ptx::ldg_here_s32(p.expert_ids + x.m_tile);
    if (p.skip_padding) {
      const int32_t* id = p.sorted_ids + (int64_t)x.m_tile * BM;
      x.id1 = ptx::ldg_here_s32(id + 32), x.id2 = ptx::ldg_here_s32(id + 64), x.id3 = ptx::ldg_here_s32(id + 96);
    }
  }
  return x;
}

// A unit of work = one output tile x one K range.  Dense problems number their units: the tiles
// [0, full_units) whole, then `splits` consecutive units per remaining tile.
struct Unit {
  int tile, kb_begin, kb_stop;
  int slot;  // split units: which [BM][BN] float32 block of the partial-sum scratch
  bool split;
};
template <Form kForm>
__device__ __forceinline__ Unit decode_unit(const GemmParams& p, int u) {
  constexpr bool kGrouped = kForm == Form::kGrouped || kForm == Form::kActivated;
  Unit x;
  x.slot = 0;
  if constexpr (kForm == Form::kSplit) {  // CTA `rank` of a cluster of p.splits: that part of the tile's slabs
    x.tile = u / p.splits, x.split = true;
    const int rank = u - x.tile * p.splits;
    x.kb_begin = rank * p.kb_total / p.splits, x.kb_stop = (rank + 1) * p.kb_total / p.splits;
    return x;
  }
  if (!kGrouped && p.sk_share > 0) {
    // unit u = piece u / sk_ctas of the run of CTA u % sk_ctas
    const int piece = u / p.sk_ctas, c = u - piece * p.sk_ctas;
    const int lo = c * p.sk_share, hi = min(lo + p.sk_share, p.sk_total);
    const int t0 = lo / p.kb_total;
    x.tile = t0 + piece, x.slot = u, x.split = true;
    // the run restricted to the slabs of tile t0 + piece (empty ranges are skipped by every role)
    const int tb = x.tile * p.kb_total;
    x.kb_begin = max(lo, tb) - tb;
    x.kb_stop = max(min(hi, tb + p.kb_total) - tb, x.kb_begin);
    return x;
  }
  if (kGrouped || u < p.full_units) {
    x.tile = u, x.kb_begin = 0, x.kb_stop = p.kb_total, x.split = false;
  } else {
    const int v = u - p.full_units;
    x.tile = p.full_units + v / p.splits;
    const int sp = v - (x.tile - p.full_units) * p.splits;
    x.kb_begin = sp * p.kb_per_split;
    x.kb_stop = min(p.kb_total, x.kb_begin + p.kb_per_split);
    x.slot = v;
    x.split = true;
  }
  return x;
}

// Epilogue of the activated form for one row: acc holds 64 gate and 64 up values, columns cgrp * 64 .. of group `n_tile`.
// Rounded to T as a stored product would be, silu(gate) rounded to T, times up rounded to T, then the quantizer: the
// arithmetic of silu_mul_quant_kernel, bit for bit.  The other half of the group is in the same lane of the other warp of
// the quadrant, so the two warps exchange their maxima; `half` is this row's place of column group 0.  False when the wait
// for the other warp expired.  The 64 codes come back in `codes`.
template <typename T>
__device__ __forceinline__ bool activate_row(const GemmParams& p, const float (&acc)[128], int cgrp, float2* half, uint32_t bar,
                                             uint32_t parity, uint4 (&codes)[4], float& scale) {
  constexpr float kEps = 1e-10f;  // as the quantizer of the layer's activations
  uint4 h[8];
  uint32_t top = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 8 * j + 2 * k;
      float g[2];
      Packed2<T>::unpack(Packed2<T>::pack(acc[c], acc[c + 1]), g);
      w[k] = Packed2<T>::round_mul(silu_f32(g[0]), silu_f32(g[1]), Packed2<T>::pack(acc[64 + c], acc[64 + c + 1]));
      top = Packed2<T>::max_abs_nan(top, w[k]);
    }
    h[j] = make_uint4(w[0], w[1], w[2], w[3]);
  }
  float t2[2];
  Packed2<T>::unpack(top, t2);
  float most = max3_abs_nan(kEps, t2[0], t2[1]), finite = most;  // (finite: the maximum of what is a number)
  if (most != most) {
    finite = kEps;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v[8];
      unpack_chunk<T>(h[j], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) finite = fmaxf(finite, fabsf(v[k]));
    }
  }
  ptx::sts_64(ptx::smem_u32(half + cgrp * BM), __float_as_uint(most), __float_as_uint(finite));
  __syncwarp();
  ptx::mbar_arrive_if(bar, (threadIdx.x & 31) == 0);
  if (!SGLB_WAIT(bar, parity)) return false;
  const float2 other = ptx::lds_f32x2(ptx::smem_u32(half + (cgrp ^ 1) * BM));
  most = max_nan(most, other.x), finite = fmaxf(finite, other.y);
  scale = __fdiv_rn(most, 448.0f);
  uint32_t out[8][2];
  if (most < __int_as_float(0x7f800000) && scale >= 1e-30f && scale <= 1e36f) {
    const float r = __frcp_rn(scale);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v[8];
      unpack_chunk<T>(h[j], v);
      quant_chunk_fast<T, true>(h[j], v, scale, r, -448.0f, 448.0f, out[j]);
    }
  } else {
    scale = __fdiv_rn(finite, 448.0f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v[8];
      unpack_chunk<T>(h[j], v);
      quant_chunk_careful<T>(v, scale, -448.0f, 448.0f, out[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) codes[j] = make_uint4(out[2 * j][0], out[2 * j][1], out[2 * j + 1][0], out[2 * j + 1][1]);
  return true;
}

// A tile whose K range the CTAs of a cluster have split.  CTA r owns `cluster_groups` groups of eight columns from the
// r-th on; every CTA writes the partial sums of the others' columns straight into their shared memory (of its own into the
// ring, which has been consumed), and after one barrier of the cluster each adds what it owns.  A source's sums lie as
// [owned group of eight][columns 0-3, 4-7][row][4] of float32.
template <int BN>
__host__ __device__ constexpr int cluster_groups(int splits) { return (BN / 8 + splits - 1) / splits; }
constexpr uint32_t kClusterGroupBytes = 2 * BM * 16;

// The owned columns: the sources' sums in ascending K order, bias, one rounding.  A warp takes 2 x 8 rows of 32 columns at a time.
template <int BN>
__device__ __forceinline__ void cluster_sum(const GemmParams& p, int rank, int m_tile, int n_tile, uint32_t own, uint32_t recv,
                                            int warp, int lane) {
  const int rows = (int)min((int64_t)BM, p.M - (int64_t)m_tile * BM), groups = cluster_groups<BN>(p.splits);
  const int first = rank * groups, stop = min(first + groups, BN / 8), splits = p.splits;
  const int row = warp * 8 + (lane & 7);  // and 64 further on
  const uint32_t bytes = groups * kClusterGroupBytes;
  int c8 = first + (lane >> 3), col = n_tile * BN + c8 * 8;
  uint32_t at = (uint32_t)(lane >> 3) * kClusterGroupBytes + row * 16;
  uint16_t* out = static_cast<uint16_t*>(p.C) + ((int64_t)m_tile * BM + row) * p.N + col;
  const uint16_t* bias = static_cast<const uint16_t*>(p.bias);
  for (; c8 < stop && col < p.N && row < rows; c8 += 4, col += 32, at += 4 * kClusterGroupBytes, out += 32) {  // (N: a multiple of 8)
    float a[2][8];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) a[k][j] = 0.f;
    uint32_t from = recv + at;
    for (int s = 0; s < splits; ++s) {
      const uint32_t src = s == rank ? own + at : from;
      if (s != rank) from += bytes;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 v = ptx::lds_f32x4(src + k * (64 * 16)), w = ptx::lds_f32x4(src + k * (64 * 16) + BM * 16);
        a[k][0] += v.x, a[k][1] += v.y, a[k][2] += v.z, a[k][3] += v.w;
        a[k][4] += w.x, a[k][5] += w.y, a[k][6] += w.z, a[k][7] += w.w;
      }
    }
    if (bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint16_t raw16 = __ldg(bias + col + j);
        const float b = p.out_fp16 ? __half2float(__ushort_as_half(raw16)) : __bfloat162float(__ushort_as_bfloat16(raw16));
        a[0][j] += b, a[1][j] += b;
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      uint32_t word[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(a[k][2 * j], a[k][2 * j + 1]);
        const __nv_bfloat162 b = __floats2bfloat162_rn(a[k][2 * j], a[k][2 * j + 1]);
        word[j] = p.out_fp16 ? *reinterpret_cast<const uint32_t*>(&h) : *reinterpret_cast<const uint32_t*>(&b);
      }
      if (row + 64 * k < rows) *reinterpret_cast<uint4*>(out + (int64_t)(64 * k) * p.N) = make_uint4(word[0], word[1], word[2], word[3]);
    }
  }
}

template <Form kForm, int BN_>
__global__ void __launch_bounds__(kGemmThreads, 1)
    fp8_blockscale_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                               const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_a32,
                               const GemmParams p) {
  constexpr bool kGrouped = kForm == Form::kGrouped || kForm == Form::kActivated, kAct = kForm == Form::kActivated;
  constexpr bool kEarly = kForm == Form::kOnce || kForm == Form::kSplit;  // (a CTA's first unit is known before the wait)
  static_assert(!kAct || BN_ == 256, "a tile of 128 gate and 128 up columns");
  static_assert(kForm != Form::kSplit || BN_ == 128, "partial sums beside the ring");
  using Cfg = TileCfg<BN_, kForm>;
  constexpr int BN = Cfg::BN, kStages = Cfg::kStages, kAccBufs = Cfg::kAccBufs, kAccStride = Cfg::kAccStride,
                kEpiCols = Cfg::kEpiCols, kOutGroups = Cfg::kOutGroups;
  constexpr uint32_t kStageBytes = Cfg::kStageBytes, kOutGroupBytes = Cfg::kOutGroupBytes;
  extern __shared__ uint8_t smem_raw[];
  // tiles need 1024-byte alignment for the 128-byte swizzle
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_stage = tiles + Cfg::kOutOffset;
  SharedCtl<Cfg>* ctl = reinterpret_cast<SharedCtl<Cfg>*>(tiles + Cfg::kTileArea);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctl->abort_flag;

  if constexpr (kForm == Form::kSplit) ptx::cluster_arrive();  // (a CTA's memory may be written once it runs)
  // (the reduction kernel that follows a split launch is launched programmatically: letting it be scheduled now
  // hides its launch latency; it waits for this grid to complete before it reads a partial sum)
  ptx::launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&ctl->full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->empty[s]), 1);
    }
    for (int b = 0; b < kAccBufs; ++b) {
      ptx::mbar_init(ptx::smem_u32(&ctl->tmem_full[b]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->tmem_empty[b]), kEpiWarps);
    }
    for (int d = 0; d < 2; ++d) {
      ptx::mbar_init(ptx::smem_u32(&ctl->sc_full[d]), 32);
      ptx::mbar_init(ptx::smem_u32(&ctl->sc_empty[d]), kEpiWarps);
      ptx::mbar_init(ptx::smem_u32(&ctl->desc_full[d]), 32);
      ptx::mbar_init(ptx::smem_u32(&ctl->desc_empty[d]), kEpiThreads);
    }
    ptx::mbar_init(ptx::smem_u32(&ctl->out_full), kEpiThreads);
    ptx::mbar_init(ptx::smem_u32(&ctl->out_free), 1);
    for (int i = 0; i < 4; ++i) ptx::mbar_init(ptx::smem_u32(&ctl->half_full[i]), kColGroups);
    ctl->abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&map_a);
    ptx::tma_prefetch_desc(&map_b);
    if constexpr (kEarly) {
      // The weights of the first slabs, while the quantizer before this kernel (which triggers behind its own wait, so that all
      // before it is complete) still makes the activations: 100 to 300 ns, 256 x 7168 x 2048 with it 11.16 -> 10.80 us.
      if (p.early_weights) {
        const Unit un = decode_unit<kForm>(p, blockIdx.x);
        int m_tile, n_tile;
        tile_coord(un.tile, (int)((p.M + BM - 1) / BM), p.tiles_n, p.group_m, m_tile, n_tile);
        for (int s = 0; s < min(kStages, un.kb_stop - un.kb_begin); ++s) {
          const uint32_t bar = ptx::smem_u32(&ctl->full[s]);
          ptx::mbar_arrive_expect_tx(bar, kStageBytes);
          ptx::tma_load_3d(ptx::smem_u32(tiles) + s * kStageBytes + kTileBytesA, &map_b, bar, (un.kb_begin + s) * BK, n_tile * BN, 0);
        }
      }
    }
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), kTmemCols);
    ptx::tmem_relinquish();
  }
  // (launched programmatically: the barriers and the tensor memory are set up while the kernel before this one ends;
  // nothing that it may have written is touched before the wait)
  ptx::grid_dependency_wait();
  int64_t rows = p.M;
  if (kGrouped) {
    const int64_t lim = *p.num_rows_dev;
    rows = lim < rows ? lim : rows;
  }
  const int tiles_m = (int)((rows + BM - 1) / BM);
  const int tiles_n = p.tiles_n;
  const int num_tiles = tiles_m * tiles_n;
  const int kb_total = p.kb_total;
  const int num_units = kForm == Form::kSplit ? num_tiles * p.splits
                        : kGrouped       ? num_tiles
                        : p.sk_share > 0 ? p.sk_pieces * p.sk_ctas
                                         : p.full_units + (num_tiles - p.full_units) * p.splits;
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  if constexpr (kForm == Form::kSplit) ptx::cluster_wait();
  const uint32_t tmem_base = ctl->tmem_base;
  const int64_t as_stride_k = kGrouped ? 1 : p.as_stride_k;  // (experts: dense rows)
  const bool vec_scales = as_stride_k == 1 && ((kGrouped ? kb_total : p.as_stride_m) & 3) == 0 &&
                          (reinterpret_cast<uintptr_t>(p.a_s) & 15u) == 0;
  // activation scales of slabs kb .. kb+3 of the row `a_row` points at (zero past the last slab)
  auto load_a4_row = [&](const float* a_row, int kb) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec_scales && kb + 3 < kb_total && (kb & 3) == 0) {
      v = __ldg(reinterpret_cast<const float4*>(a_row + kb));
    } else {
      if (kb + 0 < kb_total) v.x = __ldg(a_row + (int64_t)(kb + 0) * as_stride_k);
      if (kb + 1 < kb_total) v.y = __ldg(a_row + (int64_t)(kb + 1) * as_stride_k);
      if (kb + 2 < kb_total) v.z = __ldg(a_row + (int64_t)(kb + 2) * as_stride_k);
      if (kb + 3 < kb_total) v.w = __ldg(a_row + (int64_t)(kb + 3) * as_stride_k);
    }
    return v;
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    ptx::setmaxnreg_dec<Cfg::kOtherRegs>();
    if (ptx::elect_one()) {
      const uint32_t bar_empty0 = ptx::smem_u32(&ctl->empty[0]), bar_full0 = ptx::smem_u32(&ctl->full[0]);
      const uint32_t tiles0 = ptx::smem_u32(tiles);
      uint32_t s = 0, ph = 0;
      int ahead = kEarly && p.early_weights ? kStages : 0;  // slabs of the first unit whose weights are on their way
      bool alive = true;
      // With experts the next tile is looked up behind the first loads of this one: between two tiles the ring would otherwise
      // run dry for a round trip to L2.  (Dense tiles, whose coordinates are two divisions: 4096 x 32768 x 512 113.6 -> 115.9.)
      TileInfo next{};
      auto look_ahead = [&](int u) {
        if (kGrouped && u < num_units) next = tile_info<kGrouped>(p, u, tiles_m, tiles_n);
      };
      look_ahead(blockIdx.x);
      for (int u = blockIdx.x; u < num_units && alive; u += gridDim.x) {
        const Unit un = decode_unit<kForm>(p, u);
        const int kb_begin = un.kb_begin, kb_stop = un.kb_stop;
        if (kb_begin >= kb_stop) continue;  // (an empty piece of a stream-K run)
        const TileInfo at = kGrouped ? next : tile_info<kGrouped>(p, un.tile, tiles_m, tiles_n);
        const int m_tile = at.m_tile, n_tile = at.n_tile, e = at.expert;
        if (e < 0) {
          look_ahead(u + gridDim.x);
          continue;
        }
        int live = 4;
        if (kGrouped && p.skip_padding) live = at.live(p);
        // this thread shares its scheduler with promotion warps that always have work: every instruction it
        // spends per slab delays the loads, so the loop keeps only 32-bit counters that step
        const int row_a = m_tile * BM, row_b = n_tile * (kAct ? BN / 2 : BN), row_up = kAct ? (int)(p.N / 2) + row_b : 0;
        for (int k0 = kb_begin * BK; k0 < kb_stop * BK; k0 += BK) {
          if (!SGLB_WAIT(bar_empty0 + s * 8, ph ^ 1u)) { *abort_flag = 1; alive = false; break; }
          const uint32_t bar = bar_full0 + s * 8;
          const bool fetched = kEarly && ahead > 0;
          if (!fetched) ptx::mbar_arrive_expect_tx(bar, kStageBytes);
          const uint32_t dst_a = tiles0 + s * kStageBytes;
          if (!kGrouped || live == 4) {
            ptx::tma_load_2d(dst_a, &map_a, bar, k0, row_a);
          } else {  // quadrants of padding come from beyond the last row: zeros, without a byte of memory traffic
#pragma unroll
            for (int i = 0; i < 4; ++i)
              ptx::tma_load_2d(dst_a + i * (kTileBytesA / 4), &map_a32, bar, k0, i < live ? row_a + 32 * i : (int)p.M);
          }
          if (!fetched) ptx::tma_load_3d(dst_a + kTileBytesA, &map_b, bar, k0, row_b, e);
          if (kEarly) --ahead;
          if (kAct) ptx::tma_load_3d(dst_a + kTileBytesA + Cfg::kTileBytesB / 2, &map_b, bar, k0, row_up, e);
          if (kGrouped && k0 == 0) look_ahead(u + gridDim.x);
          if (++s == (uint32_t)kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        ahead = 0;
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    ptx::setmaxnreg_dec<Cfg::kOtherRegs>();
    if (ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::make_idesc_e4m3_f32(BM, BN);
      // Operand descriptor (K-major, 128-byte swizzle): low word = address/16 | LBO(1) << 16, high word =
      // SBO(1024/16) | version 1 (bit 46) | layout SWIZZLE_128B (2 at bit 61).  Only the low word changes.
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
      const uint32_t desc_lo0 = ((ptx::smem_u32(tiles) & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t bar_full0 = ptx::smem_u32(&ctl->full[0]), bar_empty0 = ptx::smem_u32(&ctl->empty[0]);
      const uint32_t bar_tfull0 = ptx::smem_u32(&ctl->tmem_full[0]), bar_tempty0 = ptx::smem_u32(&ctl->tmem_empty[0]);
      uint32_t s = 0, ph = 0, aph = 0;  // aph: phase of every accumulator buffer, one bit each
      bool alive = true;
      // (whether a tile has an expert is asked a unit ahead: the answer is a round trip to L2)
      auto expert_of = [&](int u) -> int {
        if (!kGrouped || u >= num_units) return 0;
        int m_tile, n_tile;
        tile_coord(u, tiles_m, tiles_n, p.group_m, m_tile, n_tile);
        return ptx::ldg_here_s32(p.expert_ids + m_tile);
      };
      int e_next = expert_of(blockIdx.x);
      for (int u = blockIdx.x; u < num_units && alive; u += gridDim.x) {
        const Unit un = decode_unit<kForm>(p, u);
        const int kb_begin = un.kb_begin, kb_stop = un.kb_stop, e = e_next;
        e_next = expert_of(u + gridDim.x);
        if (kb_begin >= kb_stop || e < 0) continue;
        uint32_t buf = 0;  // (every unit starts with buffer 0, as the promotion does)
        for (int kb = kb_begin; kb < kb_stop; ++kb) {
          // (the buffer last: it is what the MMAs wait for, and a wait that finds its barrier ready takes 80 clocks too)
          if (!SGLB_WAIT(bar_full0 + s * 8, ph)) { *abort_flag = 1; alive = false; break; }
          if (!SGLB_WAIT(bar_tempty0 + buf * 8, ((aph >> buf) & 1u) ^ 1u)) { *abort_flag = 1; alive = false; break; }
          ptx::tc_fence_after();
          const uint32_t a_lo = desc_lo0 + s * (kStageBytes >> 4);
          const uint32_t b_lo = a_lo + (kTileBytesA >> 4);
          const uint32_t d_tmem = tmem_base + buf * kAccStride;
#pragma unroll
          for (int k = 0; k < BK / 32; ++k) {
            // advancing 32 bytes along K inside the 128-byte swizzled row = +2 in the descriptor's 16-byte units
            ptx::mma_f8f6f4(d_tmem, ptx::pack_f32x2(a_lo + 2 * k, kDescHi), ptx::pack_f32x2(b_lo + 2 * k, kDescHi), idesc,
                            k > 0 ? 1u : 0u);
          }
          ptx::mma_commit(bar_empty0 + s * 8);
          ptx::mma_commit(bar_tfull0 + buf * 8);
          if (++s == (uint32_t)kStages) {
            s = 0;
            ph ^= 1u;
          }
          aph ^= 1u << buf;
          buf = buf + 1 == (uint32_t)kAccBufs ? 0u : buf + 1;
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------ output stores ------------------------------
    ptx::setmaxnreg_dec<Cfg::kOtherRegs>();
    // One thread hands every finished tile to the TMA engine: it waits until all promotion threads have parked their
    // part of the tile in the staging area, issues the stores, waits until they have read the staging and gives it
    // back.  The promotion warps never wait for each other or for a store to be issued: each goes on to its next
    // unit as soon as its own part is parked.
    if (p.tma_out && ptx::elect_one()) {
      const uint32_t bar_out_full = ptx::smem_u32(&ctl->out_full), bar_out_free = ptx::smem_u32(&ctl->out_free);
      uint32_t oph = 0;
      for (int u = blockIdx.x; u < num_units; u += gridDim.x) {
        const Unit un = decode_unit<kForm>(p, u);
        if (un.kb_begin >= un.kb_stop || un.split) continue;
        if (!SGLB_WAIT(bar_out_full, oph)) {
          *abort_flag = 1;
          break;
        }
        oph ^= 1u;
        if (*abort_flag == 0) {  // (after a give-up the tile is incomplete: nothing is stored)
          int m_tile, n_tile;
          tile_coord(un.tile, tiles_m, tiles_n, p.group_m, m_tile, n_tile);
          const int n_end = (int)min((int64_t)n_tile * BN + BN, p.N);
          const CUtensorMap* cmap = &map_c;
          int out_row0 = m_tile * BM;
          if (p.push_maps != nullptr) {
            const int owner = out_row0 / p.push_rows_per_owner;
            cmap = p.push_maps + owner;
            out_row0 += (p.push_rank - owner) * p.push_rows_per_owner;
          }
          if constexpr (kAct) {
            const int live = p.skip_padding ? live_quadrants(p, m_tile) : 4;
            for (int i = 0; i < live; ++i)
              ptx::tma_store_2d(cmap, ptx::smem_u32(out_stage) + i * (32 * 128), n_tile * 128, out_row0 + 32 * i);
          } else {
            // (with padding to skip, the map's box is a quadrant)
            const int parts = kGrouped && p.skip_padding ? live_quadrants(p, m_tile) : 1;
#pragma unroll
            for (int g = 0; g < kOutGroups; ++g) {
              if (n_tile * BN + g * 64 < n_end)
                for (int i = 0; i < parts; ++i)
                  ptx::tma_store_2d(cmap, ptx::smem_u32(out_stage) + g * kOutGroupBytes + i * (32 * 128), n_tile * BN + g * 64,
                                    out_row0 + 32 * i);
            }
          }
          ptx::tma_store_commit();
        }
        ptx::tma_store_wait_read();
        ptx::mbar_arrive(bar_out_free);
      }
      // tiles pushed to other GPUs have landed before the kernel counts as finished
      if (p.push_maps != nullptr) ptx::tma_store_wait_all();
    }
  } else if (warp == 3) {
    // ------------------------------ unit scout ------------------------------
    ptx::setmaxnreg_dec<Cfg::kOtherRegs>();
    // Walks the CTA's units ahead of the promotion warps: a descriptor of each in one of two slots (every unit, empty
    // stream-K pieces included, so that the two sides count alike), then the products of activation and weight-block
    // scales of its slabs, four slabs per slot of a two-slot ring.  The promotion warps then touch no global memory and
    // read shared memory once in four slabs, a slab ahead of the use (an access takes a hundred clocks and more beside
    // the MMA's operand reads; scales read slab by slab cost 10 % of the rate).  All 32 lanes probe the same barrier
    // word, so the outcome of a wait is uniform.
    const uint32_t bar_dfull0 = ptx::smem_u32(&ctl->desc_full[0]), bar_dempty0 = ptx::smem_u32(&ctl->desc_empty[0]);
    const uint32_t bar_sfull0 = ptx::smem_u32(&ctl->sc_full[0]), bar_sempty0 = ptx::smem_u32(&ctl->sc_empty[0]);
    uint32_t ds = 0, dph = 0, ss = 0, sph = 0;
    bool alive = true;
    // With experts a tile's ids are asked for a tile ahead, and the scales of its rows all at once: looked up one after the
    // other, its expert, its rows' ids, their weights and two halves of the scales, twice, took as long as a tile of six slabs,
    // and the promotion warps waited 2 500 to 3 600 of 9 000 clocks a tile for them (dense: 410 in all before the first slab;
    // so 750).  Second product of 131072 rows through 128 experts of 2048 x 768: 393 -> 334 us, layer 1 219 -> 1 148.
    constexpr int kRowsAhead = kForm == Form::kGrouped ? 4 : 2;  // (the others have no registers left for four)
    const bool sorted_weights = kForm == Form::kGrouped && p.tma_out && p.row_weights != nullptr;
    TileInfo next{};
    int next_id[4] = {0, 0, 0, 0};
    auto look_ahead = [&](int u) {
      if (!kGrouped || u >= num_units) return;
      next = tile_info<kGrouped>(p, u, tiles_m, tiles_n);
      if (sorted_weights) {
#pragma unroll
        for (int k = 0; k < 4; ++k) next_id[k] = ptx::ldg_here_s32(p.sorted_ids + (int64_t)next.m_tile * BM + 32 * k + lane);
      }
    };
    look_ahead(blockIdx.x);
    for (int u = blockIdx.x; u < num_units && alive; u += gridDim.x) {
      if (!SGLB_WAIT(bar_dempty0 + ds * 8, dph ^ 1u)) {
        *abort_flag = 1;
        break;
      }
      const Unit un = decode_unit<kForm>(p, u);
      UnitDesc* d = &ctl->desc[ds];
      int m_tile = 0, n_tile = 0, e = 0, live = 4;
      const bool work = un.kb_begin < un.kb_stop;
      if (kGrouped) {
        m_tile = next.m_tile, n_tile = next.n_tile, e = next.expert;
        if (p.skip_padding) live = next.live(p);
      } else if (work) {
        tile_coord(un.tile, tiles_m, tiles_n, p.group_m, m_tile, n_tile);
      }
      if (lane == 0) {
        d->m_tile = m_tile, d->n_tile = n_tile, d->expert = e, d->kb_begin = un.kb_begin;
        d->kb_stop = un.kb_stop, d->split = un.split ? 1 : 0, d->slot = un.slot, d->live = live;
      }
      float row_w[4];  // (stored with the tile's first scales, which the promotion warps wait for as well)
      float* row_w_at = &ctl->row_w[ds][0];
      if (sorted_weights) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          row_w[k] = next_id[k] >= 0 && next_id[k] < p.numel ? ptx::ldg_here_f32(p.row_weights + next_id[k]) : 0.f;
      }
      ptx::mbar_arrive(bar_dfull0 + ds * 8);  // every lane: its own writes are released with its arrival
      look_ahead(u + gridDim.x);
      if (++ds == 2u) {
        ds = 0;
        dph ^= 1u;
      }
      if (!work || e < 0) continue;
      const int nb_tile = kAct ? n_tile : min(n_tile * BN / kScaleBlockN, p.nb_total - 1);
      const int nb_next = kAct ? p.nb_total / 2 + n_tile : min(nb_tile + 1, p.nb_total - 1);
      const float* b_row0 = p.b_s + ((int64_t)e * p.nb_total + nb_tile) * kb_total;
      const float* b_row1 = p.b_s + ((int64_t)e * p.nb_total + nb_next) * kb_total;
      for (int kb = un.kb_begin; kb < un.kb_stop; kb += kScSlabs) {
        // The scales of the tile's weight blocks: with experts, where registers are short, lanes 0-3 hold those of the first block
        // and lanes 4-7 of the second (a short dense product waits 0.15 us longer for its first ones so).
        float bv = 0.f, bl[2][kScSlabs];
        if (kGrouped) {
          if (lane < (BN > kScaleBlockN ? 2 : 1) * kScSlabs && kb + (lane & 3) < kb_total)
            bv = __ldg((lane < kScSlabs ? b_row0 : b_row1) + kb + (lane & 3));
        } else {
#pragma unroll
          for (int j = 0; j < kScSlabs; ++j) {
            bl[0][j] = kb + j < kb_total ? __ldg(b_row0 + kb + j) : 0.f;
            bl[1][j] = BN > kScaleBlockN && kb + j < kb_total ? __ldg(b_row1 + kb + j) : 0.f;
          }
        }
        const uint32_t sc_addr = ptx::smem_u32(&ctl->sc[ss][0][lane][0]);
#pragma unroll
        for (int half = 0; half < 4 / kRowsAhead; ++half) {
          float4 av[kRowsAhead];
#pragma unroll
          for (int k = 0; k < kRowsAhead; ++k) {
            // (the last tile's rows past M, of which a_s has none, read the last row's scales and are never stored)
            const int row = min(m_tile * BM + lane + 32 * (kRowsAhead * half + k), (int)p.M - 1);
            av[k] = load_a4_row(p.a_s + (kGrouped ? (int64_t)((uint64_t)(uint32_t)row * (uint32_t)kb_total) : row * p.as_stride_m), kb);
          }
          if (half == 0 && !SGLB_WAIT(bar_sempty0 + ss * 8, sph ^ 1u)) {
            *abort_flag = 1;
            alive = false;
            break;
          }
          if (half == 0 && kb == 0 && sorted_weights) {
#pragma unroll
            for (int k = 0; k < 4; ++k) row_w_at[32 * k + lane] = row_w[k];
          }
#pragma unroll
          for (int w = 0; w < (BN > kScaleBlockN ? 2 : 1); ++w) {
            float b[kScSlabs];
#pragma unroll
            for (int j = 0; j < kScSlabs; ++j) b[j] = kGrouped ? __shfl_sync(0xffffffffu, bv, kScSlabs * w + j) : bl[w][j];
#pragma unroll
            for (int k = 0; k < kRowsAhead; ++k)
              ptx::sts_128(sc_addr + w * (BM * 16) + (kRowsAhead * half + k) * (32 * 16),
                           make_uint4(__float_as_uint(av[k].x * b[0]), __float_as_uint(av[k].y * b[1]), __float_as_uint(av[k].z * b[2]),
                                      __float_as_uint(av[k].w * b[3])));
          }
        }
        if (!alive) break;
        ptx::mbar_arrive(bar_sfull0 + ss * 8);
        if (++ss == 2u) {
          ss = 0;
          sph ^= 1u;
        }
      }
    }
  } else if (warp >= kEpiWarp0) {
    // ------------------------------ promotion + epilogue ------------------------------
    ptx::setmaxnreg_inc<Cfg::kPromoRegs>();
    // A warp whose wait expires leaves its loops; the other roles then sit out their own limits.
    const int q = warp & 3;                     // TMEM lane quadrant this warp may read
    const int cgrp = (warp - kEpiWarp0) >> 2;   // column group: columns cgrp*kEpiCols .. of the tile
    constexpr int kPiecesMax = kEpiCols / 32;
    const int row_in_tile = q * 32 + lane;
    const uint32_t bar_tfull0 = ptx::smem_u32(&ctl->tmem_full[0]), bar_tempty0 = ptx::smem_u32(&ctl->tmem_empty[0]);
    // (activated form: a warp's columns are cgrp * 64 .. of the gate half and the same of the up half)
    const uint32_t taddr0 = tmem_base + ((uint32_t)(q * 32) << 16) + cgrp * (kAct ? kEpiCols / 2 : kEpiCols);
    constexpr int kPiece2 = kAct ? BN / 2 : 64;  // TMEM columns from a warp's first to its 64th
    const uint32_t bar_out_full = ptx::smem_u32(&ctl->out_full), bar_out_free = ptx::smem_u32(&ctl->out_free);
    const uint32_t bar_dfull0 = ptx::smem_u32(&ctl->desc_full[0]), bar_dempty0 = ptx::smem_u32(&ctl->desc_empty[0]);
    const uint32_t desc_addr0 = ptx::smem_u32(&ctl->desc[0]);
    const uint32_t bar_sfull0 = ptx::smem_u32(&ctl->sc_full[0]), bar_sempty0 = ptx::smem_u32(&ctl->sc_empty[0]);
    SGLB_MBAR_ASK_DECL();
    uint32_t oph = 0, ds = 0, dph = 0, ss = 0, sph = 0, half_ph = 0;
    uint32_t aph[kAccBufs];  // phase of every accumulator buffer
#pragma unroll
    for (int b = 0; b < kAccBufs; ++b) aph[b] = 0;
#ifdef SGLB_TRACE
    int trace_unit = -1;
#endif
    for (int u = blockIdx.x; u < num_units; u += gridDim.x) {
#ifdef SGLB_TRACE
      ++trace_unit;
#endif
      SGLB_STAMP(0);
      // the unit as the scout warp described it (without a descriptor there is nothing to walk: leave)
      if (!SGLB_WAIT(bar_dfull0 + ds * 8, dph)) {
        *abort_flag = 1;
        break;
      }
      const uint32_t desc_addr = desc_addr0 + ds * (uint32_t)sizeof(UnitDesc);
      // the descriptor is handed back (by every thread) once nothing more is read from it
      auto release_desc = [&]() {
        ptx::mbar_arrive(bar_dempty0 + ds * 8);
        if (++ds == 2u) {
          ds = 0;
          dph ^= 1u;
        }
      };
      const float4 h0 = ptx::lds_f32x4(desc_addr + (uint32_t)offsetof(UnitDesc, m_tile));
      const int m_tile = __float_as_int(h0.x), n_tile = __float_as_int(h0.y), kb_begin = __float_as_int(h0.w);
      const int kb_stop = __float_as_int(ptx::lds_f32(desc_addr + (uint32_t)offsetof(UnitDesc, kb_stop)));
      if (kb_begin >= kb_stop) {  // (an empty piece of a stream-K run; uniform over the CTA)
        release_desc();
        continue;
      }
      if (kGrouped && q >= __float_as_int(ptx::lds_f32(desc_addr + (uint32_t)offsetof(UnitDesc, live)))) {
        // None of this warp's rows counts: it hands everything on unread and stores nothing.  About 128 rows an expert, of
        // which every second one then has a second tile with a few rows (32768 rows, 256 experts of 7168 x 2048, sustained):
        // layer 3 491 -> 3 405 us, mostly by the power that the other warps and the MMAs (zeros) no longer share.  In dense
        // products, which have one such row of tiles, the test cost more than it gave (4096 x 36864 x 7168 1 036 -> 1 041).
        int left = __float_as_int(h0.z) < 0 ? 0 : kb_stop - kb_begin;
        release_desc();
        bool ok = true;
        for (; left > 0 && ok; left -= 4) {
          ok = SGLB_WAIT(bar_sfull0 + ss * 8, sph);
          if (ok) ptx::mbar_arrive_if(bar_sempty0 + ss * 8, lane == 0);
          ss ^= 1u;
          sph ^= ss == 0 ? 1u : 0u;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int b = i % kAccBufs;
            if (i < left && ok) {
              ok = SGLB_WAIT(bar_tfull0 + b * 8, aph[b]);
              aph[b] ^= 1u;
              if (ok) ptx::mbar_arrive_if(bar_tempty0 + b * 8, lane == 0);
            }
          }
        }
        if (ok && p.tma_out) {  // (the staging area takes part in turn, so that no arrival counts for the tile before)
          ok = SGLB_WAIT(bar_out_free, oph ^ 1u);
          oph ^= 1u;
          if (ok) ptx::mbar_arrive(bar_out_full);
        }
        if (!ok) {
          *abort_flag = 1;
          break;
        }
        continue;
      }
      const int64_t row = (int64_t)m_tile * BM + row_in_tile;
      const int n0 = n_tile * BN + cgrp * kEpiCols;            // first of this warp's columns
      const int n_end = (int)min((int64_t)n_tile * BN + BN, p.N);  // one past the tile's last valid column
      const int e = kGrouped ? __float_as_int(h0.z) : 0;
      float acc[kEpiCols];
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j) acc[j] = 0.f;
      if (e >= 0) {
        // Scales of four slabs at a time from the scout's ring, requested a slab ahead.  A warp's columns lie in one weight
        // block; columns wholly past N take the last block's.
        static_assert(kScaleBlockN % kEpiCols == 0 && kAccBufs <= 4 && 4 % kAccBufs == 0, "one weight block per warp");
        const bool second = !kAct && BN > kScaleBlockN && n0 / kScaleBlockN != n_tile * BN / kScaleBlockN && n0 / kScaleBlockN < p.nb_total;
        const uint32_t sc_addr0 = ptx::smem_u32(&ctl->sc[0][0][row_in_tile][0]) + (second ? BM * 16 : 0);
        float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f), s4_up = s4;
        auto fetch_scales = [&]() -> bool {
          if (!SGLB_WAIT(bar_sfull0 + ss * 8, sph)) return false;
          s4 = ptx::lds_f32x4(sc_addr0 + ss * (Cfg::kScBlocks * BM * 16));
          if (kAct) s4_up = ptx::lds_f32x4(sc_addr0 + ss * (Cfg::kScBlocks * BM * 16) + BM * 16);
          return true;
        };
        int left = kb_stop - kb_begin;  // slabs from the current group of four on
        bool ready = false;
        // Slab I of a group of four: the buffer, its barriers and the scale are known at compile time (with them at run
        // time a warp's bookkeeping took as many issue slots as its FMAs, each a few clocks after the one before).
        // The buffer goes back to the MMA thread as soon as its columns are in registers (one TMEM round trip per slab
        // sits on the hand-off chain MMA -> commit -> promotion -> release), then they are promoted.  Whether the next
        // slab is complete is asked before the last FMAs and looked at after them: a wait that finds its barrier ready
        // takes 50 to 100 clocks of its own.
        auto slab = [&](auto index) -> bool {
          constexpr int I = decltype(index)::value, kBuf = I % kAccBufs, kNext = (I + 1) % kAccBufs;
          // (the 32 lanes probe the same word in the same instruction, so the outcome is uniform across the
          // warp, as the warp-wide tcgen05.ld below requires)
          if (!ready && !SGLB_WAIT(bar_tfull0 + kBuf * 8, aph[kBuf])) return false;
          ptx::tc_fence_after();
          aph[kBuf] ^= 1u;
          const uint32_t taddr = taddr0 + kBuf * kAccStride;
          const float sc_lo = I == 0 ? s4.x : I == 1 ? s4.y : I == 2 ? s4.z : s4.w;
          const float sc_up = I == 0 ? s4_up.x : I == 1 ? s4_up.y : I == 2 ? s4_up.z : s4_up.w;
          auto fma = [&](int i, const uint32_t (&v)[32]) {
            const float sc = kAct && i >= 2 ? sc_up : sc_lo;
            // two columns per instruction (packed float32 FMA: the same two IEEE operations): half the issue slots
#pragma unroll
            for (int jj = 0; jj < 32; jj += 2) ptx::fma2(acc[32 * i + jj], acc[32 * i + jj + 1], v[jj], v[jj + 1], sc);
          };
          bool ok = true;
          uint32_t asked = 0;
          auto hand_back = [&]() {
            ptx::tc_fence_before();
            ptx::mbar_arrive_relaxed_if(bar_tempty0 + kBuf * 8, lane == 0);
            if (I == 0) {  // (the slot's four scales have been read: every lane's read is ordered before lane 0's release)
              __syncwarp();
              ptx::mbar_arrive_if(bar_sempty0 + ss * 8, lane == 0);
              ss ^= 1u;
              sph ^= ss == 0 ? 1u : 0u;
            }
            if (left > I + 1) {
              asked = ptx::mbar_ask(bar_tfull0 + kNext * 8, aph[kNext]);
              if (I == 3) ok = fetch_scales();
            }
          };
          uint32_t r[2][32];
          ptx::tmem_ld_32x32(taddr, r[0]);
          ptx::tmem_ld_32x32(taddr + 32, r[1]);
          ptx::tmem_ld_wait();
          if constexpr (kPiecesMax == 2) {
            hand_back();
            fma(0, r[0]);
            fma(1, r[1]);
          } else {  // (128 accumulators leave room for two pieces at a time)
            fma(0, r[0]);
            ptx::tmem_ld_32x32(taddr + kPiece2, r[0]);
            fma(1, r[1]);
            ptx::tmem_ld_32x32(taddr + kPiece2 + 32, r[1]);
            ptx::tmem_ld_wait();
            hand_back();
            fma(2, r[0]);
            fma(3, r[1]);
          }
          ready = ptx::mbar_answer(asked);  // (not looked at where nothing was asked: the unit ends)
          return ok;
        };
        bool ok = fetch_scales();
        SGLB_STAMP(1);
        while (ok && left > 0) {
          ok = slab(std::integral_constant<int, 0>{}) && (left < 2 || slab(std::integral_constant<int, 1>{})) &&
               (left < 3 || slab(std::integral_constant<int, 2>{})) && (left < 4 || slab(std::integral_constant<int, 3>{}));
          left -= 4;
        }
        if (!ok) {
          *abort_flag = 1;
          break;
        }
      }
      // (whether the unit is a piece of a split tile, and its slot among the partial sums, are read only now: two
      // registers fewer across the slab loop)
      Unit un;
      {
        const float4 h1 = ptx::lds_f32x4(desc_addr + (uint32_t)offsetof(UnitDesc, kb_stop));
        un.tile = 0, un.kb_begin = kb_begin, un.kb_stop = kb_stop;
        un.split = __float_as_int(h1.y) != 0, un.slot = __float_as_int(h1.z);
      }
      if constexpr (kForm == Form::kGrouped) {
        if (e >= 0 && p.tma_out && p.row_weights != nullptr) {  // (rows of no expert stay zero, and have no weights there)
          const float w = ptx::lds_f32(ptx::smem_u32(&ctl->row_w[ds][row_in_tile]));
#pragma unroll
          for (int j = 0; j < kEpiCols; ++j) acc[j] *= w;
        }
      }
      release_desc();
      // ---- store ----
      SGLB_STAMP(2);
      if (un.split) {
        // this unit's float32 partial sums, tile-local layout; a second kernel adds the units of a tile in a
        // fixed order, adds the bias and rounds once
        if (kForm == Form::kSplit) {
          if (row < rows) {
            const int rank = (int)blockIdx.x % p.splits, groups = cluster_groups<BN>(p.splits), c0 = cgrp * (kEpiCols / 8);
            int owner = c0 / groups, idx = c0 - owner * groups;
            const uint32_t own = ptx::smem_u32(tiles) + row_in_tile * 16, bytes = groups * kClusterGroupBytes;
            const uint32_t before = ptx::smem_u32(out_stage) + row_in_tile * 16 + (rank - 1) * bytes, after = before + bytes;
#pragma unroll
            for (int j = 0; j < kEpiCols / 8; ++j) {
              const float* a = acc + 8 * j;
              // (to CTAs of lower rank this one is source rank - 1 of the others')
              const uint32_t to = ptx::cluster_map((owner == rank ? own : owner < rank ? before : after) + idx * kClusterGroupBytes, owner);
              ptx::sts_cluster_f32x4(to, a[0], a[1], a[2], a[3]);
              ptx::sts_cluster_f32x4(to + BM * 16, a[4], a[5], a[6], a[7]);
              if (++idx == groups) idx = 0, ++owner;
            }
          }
        } else if (row < rows) {  // (rows past M are never read back)
          // [column / 4][row][4]: the 32 lanes of a warp (32 consecutive rows) write 512 contiguous bytes per store.
          float* dst = p.partial + (int64_t)un.slot * (BM * BN) + ((int64_t)(cgrp * kEpiCols / 4) * BM + row_in_tile) * 4;
#pragma unroll
          for (int j = 0; j < kEpiCols / 4; ++j)
            *reinterpret_cast<float4*>(dst + (int64_t)j * BM * 4) =
                make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
        }
        continue;
      }
      if constexpr (kAct) {  // codes of this row's half group into the staging area (128-byte rows, swizzled), as below
        const uint32_t bar_half = ptx::smem_u32(&ctl->half_full[q]);
        float2* half = &ctl->half_max[half_ph][0][row_in_tile];
        uint4 codes[4];
        float scale;
        if (!(p.out_fp16 ? activate_row<__half>(p, acc, cgrp, half, bar_half, half_ph, codes, scale)
                         : activate_row<__nv_bfloat16>(p, acc, cgrp, half, bar_half, half_ph, codes, scale)) ||
            !SGLB_WAIT(bar_out_free, oph ^ 1u)) {
          *abort_flag = 1;
          break;
        }
        oph ^= 1u;
        const uint32_t stage = ptx::smem_u32(out_stage) + row_in_tile * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) ptx::sts_128(stage + (((cgrp * 4 + j) ^ (row_in_tile & 7)) << 4), codes[j]);
        if (cgrp == 0 && row < rows) p.act_s[row * (p.N / 256) + n_tile] = scale;
        ptx::fence_async_smem();
        ptx::mbar_arrive(bar_out_full);
        half_ph ^= 1u;
        continue;
      }
      if (!kGrouped || p.tma_out) {  // (dense tiles always leave this way)
        // Rows of C are contiguous: round to the output type, park the warp's 32 x 64 block in shared memory
        // (128-byte rows, 16-byte chunks XOR-swizzled by the row so that the 32 lanes of a store spread over
        // all banks); the storing thread (warp 2) hands the 128 x 64 blocks to the TMA engine, which clips them to
        // the tensor.  The store drains while the next tile is being promoted.
        // The staging area is free once the stores of the previous tile have read it.
        if (!SGLB_WAIT(bar_out_free, oph ^ 1u)) {
          *abort_flag = 1;
          break;
        }
        oph ^= 1u;
        SGLB_STAMP(3);
        if (n0 < n_end) {
          if (p.bias != nullptr) {
            // (tile columns past N are clipped by the store; their bias reads are clamped to stay in bounds)
            const uint16_t* bsrc = static_cast<const uint16_t*>(p.bias);
#pragma unroll
            for (int j = 0; j < kEpiCols; ++j) {
              const uint16_t raw16 = __ldg(bsrc + min(n0 + j, (int)p.N - 1));
              acc[j] += p.out_fp16 ? __half2float(__ushort_as_half(raw16)) : __bfloat162float(__ushort_as_bfloat16(raw16));
            }
          }
          // round pairs of adjacent columns with one packed conversion each, and store every eight as they are rounded, so
          // that conversions and shared-memory stores overlap (K = 512, where a tile is four slabs: 4096 x 32768 114.8 us
          // with all of the row rounded first, 113.1 so; long K equal)
          const uint32_t stage0 = ptx::smem_u32(out_stage) + row_in_tile * 128;
          const uint32_t swz = (uint32_t)(row_in_tile & 7);
          auto park = [&](auto round2) {
#pragma unroll
            for (int j = 0; j < kEpiCols / 8; ++j) {
              const int col = cgrp * kEpiCols + j * 8;  // within the tile: 64-column group col / 64, 16-byte chunk (col % 64) / 8
              const float* a = acc + 8 * j;
              ptx::sts_128(stage0 + (col >> 6) * kOutGroupBytes + ((((col & 63) >> 3) ^ swz) << 4),
                           make_uint4(round2(a[0], a[1]), round2(a[2], a[3]), round2(a[4], a[5]), round2(a[6], a[7])));
            }
          };
          if (p.out_fp16)
            park([](float x, float y) {
              const __half2 h = __floats2half2_rn(x, y);
              return *reinterpret_cast<const uint32_t*>(&h);
            });
          else
            park([](float x, float y) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
              return *reinterpret_cast<const uint32_t*>(&h);
            });
          ptx::fence_async_smem();  // this thread's part is visible to the TMA engine before it arrives
        }
        SGLB_STAMP(4);
        ptx::mbar_arrive(bar_out_full);
        SGLB_STAMP(5);
        SGLB_STAMP(6);
        continue;
      }
      // Grouped scatter: the rows go to the token-major slots that sorted_token_ids names.  Through this warp's part of the
      // staging area (same layout), so that every store instruction writes 128 contiguous bytes of four rows; stored
      // row by row from the accumulators, each lane wrote 16 bytes of its own row at a time, half a sector.
      if constexpr (kForm == Form::kGrouped) {
        int dst = -1;
        if (row < rows) {
          const int32_t id = p.sorted_ids[row];
          if (id >= 0 && id < p.numel) {
            dst = id;
            if (p.row_weights != nullptr) {
              const float w = __ldg(p.row_weights + id);
#pragma unroll
              for (int j = 0; j < kEpiCols; ++j) acc[j] *= w;
            }
          }
        }
        const uint32_t stage0 = ptx::smem_u32(out_stage) + cgrp * (kEpiCols / 64) * kOutGroupBytes + q * 32 * 128;
#pragma unroll
        for (int g = 0; g < kEpiCols / 64; ++g) {
          const uint32_t stage = stage0 + g * kOutGroupBytes;
          __syncwarp();  // the part has been read
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint32_t word[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float v0 = acc[g * 64 + j * 8 + 2 * k], v1 = acc[g * 64 + j * 8 + 2 * k + 1];
              if (p.out_fp16) {
                const __half2 o = __floats2half2_rn(v0, v1);
                word[k] = *reinterpret_cast<const uint32_t*>(&o);
              } else {
                const __nv_bfloat162 o = __floats2bfloat162_rn(v0, v1);
                word[k] = *reinterpret_cast<const uint32_t*>(&o);
              }
            }
            ptx::sts_128(stage + lane * 128 + ((j ^ (lane & 7)) << 4), make_uint4(word[0], word[1], word[2], word[3]));
          }
          __syncwarp();
          const int piece = lane & 7, n = n0 + g * 64 + piece * 8;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r4 = k * 4 + (lane >> 3), to = __shfl_sync(0xffffffffu, dst, r4);
            const uint4 v = ptx::lds_128(stage + r4 * 128 + ((piece ^ (r4 & 7)) << 4));
            if (to >= 0 && n < n_end) *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.C) + (int64_t)to * p.N + n) = v;
          }
        }
      }
    }
  }

  // ------------------------------ sum over the CTAs of the cluster ------------------------------
  if constexpr (kForm == Form::kSplit) {
    __syncwarp();
    ptx::cluster_sync();  // (nobody touches another CTA's memory after it)
    if (warp >= kEpiWarp0 && ctl->abort_flag == 0) {
      const int tile = blockIdx.x / p.splits;
      int m_tile, n_tile;
      tile_coord(tile, tiles_m, tiles_n, p.group_m, m_tile, n_tile);
      cluster_sum<BN>(p, (int)blockIdx.x - tile * p.splits, m_tile, n_tile, ptx::smem_u32(tiles), ptx::smem_u32(out_stage),
                      warp - kEpiWarp0, lane);
    }
  }

  // ------------------------------ teardown ------------------------------
  // (the storing thread has waited for its last stores to read their source, in push mode to land, before it
  // reaches the barrier below)
  ptx::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag != 0 && threadIdx.x == 0) {
    atomicExch(&g_gemm_status, 1);
    // give TMA copies that may still be in flight time to land before the CTA's shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Thread i of a tile's reduction -> (row, first of 8 columns), rows fastest, so that neighbouring threads read neighbouring
// words of a unit's partial sums ([column / 4][row][4]; the two halves of the eight columns lie BM float4 apart).
__device__ __forceinline__ void reduce_coord(int i, int& r, int& c8) {
  c8 = (i / BM) * 8;
  r = i % BM;
}

// Sums the partial tiles of every split output tile in ascending split order (deterministic), adds the bias,
// rounds once and writes the part of the tile that lies inside C.  One thread per 8 consecutive columns of a row;
// grid = (split tiles, BM * BN / 8 / 256).
template <typename OutT>
__global__ void __launch_bounds__(256)
    split_reduce_kernel(const float* __restrict__ partial, OutT* __restrict__ C, const OutT* __restrict__ bias,
                        int64_t M, int64_t N, int BN, int tiles_m, int tiles_n, int group_m, int full_units, int splits) {
  ptx::grid_dependency_wait();  // the GEMM's partial sums are complete and visible
  const int tile = full_units + blockIdx.x;
  int m_tile, n_tile;
  tile_coord(tile, tiles_m, tiles_n, group_m, m_tile, n_tile);
  // one thread per (row, 8-column group)
  int r, c8;
  reduce_coord(blockIdx.y * 256 + threadIdx.x, r, c8);
  const int64_t row = (int64_t)m_tile * BM + r;
  const int64_t col = (int64_t)n_tile * BN + c8;
  if (c8 >= BN || row >= M || col >= N) return;  // N is a multiple of 8: a group is inside or outside as a whole
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float4* src = reinterpret_cast<const float4*>(partial) + (int64_t)blockIdx.x * splits * (BM * BN / 4) + (c8 >> 2) * BM + r;
  for (int s = 0; s < splits; ++s, src += BM * BN / 4) {
    const float4 a = __ldg(src), b = __ldg(src + BM);
    acc[0] += a.x, acc[1] += a.y, acc[2] += a.z, acc[3] += a.w;
    acc[4] += b.x, acc[5] += b.y, acc[6] += b.z, acc[7] += b.w;
  }
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += ElemTraits<OutT>::to_f32(bias[col + j]);
  }
  uint4 raw;
  OutT* o = reinterpret_cast<OutT*>(&raw);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = ElemTraits<OutT>::from_f32(acc[j]);
  *reinterpret_cast<uint4*>(C + row * N + col) = raw;
}

// The same for stream-K runs: output tile `blockIdx.x` is the sum, in ascending K order, of the pieces of the runs
// that cover its slabs; run c covers slabs [c * share, (c + 1) * share) of the tiles x slabs space and its piece
// for this tile sits in slot c + ctas * (tile - first tile of the run).
template <typename OutT>
__global__ void __launch_bounds__(256)
    streamk_reduce_kernel(const float* __restrict__ partial, OutT* __restrict__ C, const OutT* __restrict__ bias,
                          int64_t M, int64_t N, int BN, int tiles_m, int tiles_n, int group_m, int kb_total, int share,
                          int ctas) {
  ptx::grid_dependency_wait();  // the GEMM's partial sums are complete and visible
  const int tile = blockIdx.x;
  int m_tile, n_tile;
  tile_coord(tile, tiles_m, tiles_n, group_m, m_tile, n_tile);
  int r, c8;
  reduce_coord(blockIdx.y * 256 + threadIdx.x, r, c8);
  const int64_t row = (int64_t)m_tile * BM + r;
  const int64_t col = (int64_t)n_tile * BN + c8;
  if (c8 >= BN || row >= M || col >= N) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float4* mine = reinterpret_cast<const float4*>(partial) + (c8 >> 2) * BM + r;
  const int c_first = tile * kb_total / share, c_last = ((tile + 1) * kb_total - 1) / share;
  for (int c = c_first; c <= c_last; ++c) {
    const int slot = c + ctas * (tile - c * share / kb_total);
    const float4* src = mine + (int64_t)slot * (BM * BN / 4);
    const float4 a = __ldg(src), b = __ldg(src + BM);
    acc[0] += a.x, acc[1] += a.y, acc[2] += a.z, acc[3] += a.w;
    acc[4] += b.x, acc[5] += b.y, acc[6] += b.z, acc[7] += b.w;
  }
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += ElemTraits<OutT>::to_f32(bias[col + j]);
  }
  uint4 raw;
  OutT* o = reinterpret_cast<OutT*>(&raw);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = ElemTraits<OutT>::from_f32(acc[j]);
  *reinterpret_cast<uint4*>(C + row * N + col) = raw;
}

// How a dense problem whose 128-wide tiles are more than one wave is cut into units.
//  * Fewer than two waves of tiles with a long K (256 to 512 rows or so): stream-K when its run of slabs plus the cost of the
//    partial sums is shorter than the whole waves it replaces.
//  * More tiles than SMs with a last wave that fills at most half of them: the tiles of that wave are split so
//    that the tail takes 1/splits of a tile time instead of a whole one (the other tiles are untouched).
#ifndef SGLB_TAIL_SPLIT
#define SGLB_TAIL_SPLIT 1
#endif
constexpr bool kTailSplit = SGLB_TAIL_SPLIT != 0;
#ifndef SGLB_STREAM_K
#define SGLB_STREAM_K 1
#endif
constexpr bool kStreamK = SGLB_STREAM_K != 0;
struct UnitPlan {
  int full_units, splits, kb_per_split;
  int64_t split_tiles;
  int sk_share, sk_ctas, sk_pieces;  // stream-K (sk_share > 0): supersedes the fields above
  int64_t scratch_blocks() const { return sk_share > 0 ? (int64_t)sk_pieces * sk_ctas : split_tiles * splits; }
};
static UnitPlan plan_units(int64_t M, int64_t N, int64_t K, int BN, int sms) {
  const int kb_total = (int)((K + BK - 1) / BK);
  const int64_t tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  UnitPlan pl{(int)tiles, 1, kb_total, 0, 0, 0, 2};
  int64_t s = 1, split_tiles = 0;
  if (kStreamK && tiles < 2 * sms && kb_total >= 8 && kb_total % 4 == 0) {
    // Equal runs of slabs over ALL SMs (splitting every tile the same number of ways leaves sms mod tiles of
    // them idle).
    const int64_t total = tiles * kb_total;
    int64_t share = (total + sms - 1) / sms;
    share = (share + 3) / 4 * 4;  // runs start on multiples of four slabs: aligned 128-bit loads of the activation scales
    const int64_t ctas = (total + share - 1) / share;
    const int pieces = share <= kb_total ? 2 : 3;
    bool take = false;
    if (share <= 2 * (int64_t)kb_total) {
      // Compared in slab times (about 0.45 us each): the run plus the partial sums (one piece per run and per
      // tile boundary, written and read back at about 4 TB/s, plus the second launch) against the whole waves.
      const int64_t waves = (tiles + sms - 1) / sms;
      const double partial_bytes = (double)(ctas + tiles) * BM * BN * 4 * 2;
      const double cost = (double)share + partial_bytes / 1.8e6 + 6.0;
      take = cost < 0.9 * (double)(waves * kb_total);
    }
    if (take) {
      pl.sk_share = (int)share, pl.sk_ctas = (int)ctas, pl.sk_pieces = pieces;
      return pl;
    }
  }
  if (kTailSplit && tiles > sms && kb_total >= 32) {
    const int64_t tail = tiles % sms;
    if (tail > 0 && tail * 2 <= sms) {
      s = sms / tail;
      if (s > kb_total / 8) s = kb_total / 8;
      if (s > 8) s = 8;
      split_tiles = tail;
    }
  }
  if (s > 1) {
    int per = (int)((kb_total + s - 1) / s);
    per = (per + 3) / 4 * 4;  // keeps the 128-bit loads of the activation scales aligned
    pl.splits = (kb_total + per - 1) / per;
    pl.kb_per_split = per;
    if (pl.splits > 1) {
      pl.split_tiles = split_tiles;
      pl.full_units = (int)(tiles - split_tiles);
    } else {
      pl.kb_per_split = kb_total;
    }
  }
  return pl;
}

// ---------------------------------------------------------------------------------------------
// Host side: tensor maps (encoded through the driver entry point, cached per argument tuple)
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

struct MapKey {
  const void* ptr;
  uint64_t d0, d1, d2;
  uint32_t box_rows, rank;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && box_rows == o.box_rows && rank == o.rank;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr);
    h = h * 1000003u ^ k.d0;
    h = h * 1000003u ^ k.d1;
    h = h * 1000003u ^ k.d2;
    return (h * 1000003u ^ k.box_rows) * 31u + k.rank;
  }
};

int get_tensor_map(const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t box_rows, uint32_t rank,
                          CUtensorMap* out) {
  static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{ptr, d0, d1, d2, box_rows, rank};
  auto itc = cache.find(key);
  if (itc != cache.end()) {
    *out = itc->second;
    return SGLB200_OK;
  }
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return fail(SGLB200_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {d0, d0 * d1};  // bytes (1-byte elements)
  cuuint32_t box[3] = {(cuuint32_t)BK, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(SGLB200_E_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return SGLB200_OK;
}

int get_out_map(const void* ptr, uint64_t N, uint64_t rows, int out_fp16, uint32_t box_rows, CUtensorMap* out) {
  static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{ptr, N, rows, (uint64_t)out_fp16, box_rows, 0};
  auto itc = cache.find(key);
  if (itc != cache.end()) {
    *out = itc->second;
    return SGLB200_OK;
  }
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return fail(SGLB200_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[2] = {N, rows};
  cuuint64_t strides[1] = {N * 2};
  cuuint32_t box[2] = {64u, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, out_fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                   const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(SGLB200_E_CUDA, "cuTensorMapEncodeTiled (output) failed with CUresult %d", (int)r);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return SGLB200_OK;
}

// m-tiles per rasterization group: as many as keep the group's activation rows (128*K bytes per m-tile) within
// a quarter of the L2 (measured: with half of it the streaming weight tiles start evicting the rows), in groups
// of equal size, so that the weights are read from DRAM once per group and the activations once in all.
int choose_group_m(int64_t rows, int64_t K, int tile_rows) {
  const int64_t budget = 32ll << 20;
  int64_t gmax = budget / (tile_rows * K);
  if (gmax < 2) gmax = 2;
  if (gmax < 4 && tile_rows == BM) gmax = 4;
  const int64_t tiles_m = (rows + tile_rows - 1) / tile_rows;
  const int64_t groups = (tiles_m + gmax - 1) / gmax;
  return (int)((tiles_m + groups - 1) / groups);
}

// Tile width of a dense problem (TileCfg): 128 columns where one wave of such tiles holds it.  Against 256-wide tiles that are
// split or run stream-K over all SMs, with the quantizer: 128 x 10240 x 8192 29.3 -> 24.4 us, 80 x 18432 x 7168 35.1 -> 28.9, 128 x
// 16384 x 8192 37.7 -> 32.0, 256 x 7168 x 16384 46.0 -> 44.0.  Else 256 columns where that splits K (stream-K, split tiles); else
// compared as waves x tile width, the 128-wide tile charged 156 instead of 128 (it takes 0.61 of a wide tile's time).
// `sms`: those that the launch may use.
static bool one_narrow_wave(int64_t M, int64_t N, int sms) { return ((M + BM - 1) / BM) * ((N + 127) / 128) <= sms; }
static int choose_bn(int64_t M, int64_t N, int64_t K, int sms) {
  if (one_narrow_wave(M, N, sms)) return 128;
  if (plan_units(M, N, K, 256, sms).scratch_blocks() > 0) return 256;
  const int64_t tiles_m = (M + BM - 1) / BM;
  const int64_t waves256 = (tiles_m * ((N + 255) / 256) + sms - 1) / sms;
  const int64_t waves128 = (tiles_m * ((N + 127) / 128) + sms - 1) / sms;
  return waves128 * 156 < waves256 * 256 ? 128 : 256;
}
// The expert-grouped form: rows per expert are not known on the host; with a handful of routed rows (decode) the
// 128-wide tile spreads the few row blocks over more SMs.
static int choose_bn_grouped(int64_t numel) {
  return numel <= 64 ? 128 : 256;
}

// How a dense problem runs: tile width and the cut into units.
struct DensePlan {
  int bn;
  int cluster;  // CTAs of a cluster over which every tile's slabs are split (`units` then does not count), or 1
  UnitPlan units;
  int64_t scratch_bytes() const { return cluster > 1 ? 0 : units.scratch_blocks() * (int64_t)BM * bn * (int64_t)sizeof(float); }
};
static DensePlan plan_dense(int64_t M, int64_t N, int64_t K) {
  DensePlan d;
  const int sms = sm_count();
  d.cluster = tile_splits(((M + BM - 1) / BM) * ((N + 127) / 128), (int)((K + BK - 1) / BK), M, cluster_fits());
  d.bn = d.cluster > 1 ? 128 : choose_bn(M, N, K, sms);
  // (one wave of 128-wide tiles is not cut in units of its own)
  if (one_narrow_wave(M, N, sms)) d.units = UnitPlan{(int)(((M + BM - 1) / BM) * ((N + 127) / 128)), 1, (int)((K + BK - 1) / BK), 0, 0, 0, 2};
  else d.units = plan_units(M, N, K, d.bn, sms);
  return d;
}

// Few activation rows take the kernel with the weights on the M side (gemm_rows.cu): up to 64 rows its tiles follow the
// rows there are, beyond that this kernel's 128-row tiles are at least half full.  Up to 256 rows it also takes problems of at most
// 32 tiles of 64 rows x 128 columns, of which it puts two on an SM and splits K over up to sixteen CTAs each; the weights that
// every 64 rows fetch anew come from L2.  Us of the layer, both ways: 128 rows, 512 x 7168 9.6 against 21.2 (11.3 with the K of
// 128-row tiles split over clusters), 1024 x 4096 9.5 / 14.3 (10.5), 2048 x 1024 7.7 / 8.0 (9.1); 256 rows, 512 x 2048 7.9 / 9.5
// (9.3), 1024 x 7168 12.8 / 20.7 (12.7).  Not beyond: 128 rows, 3072 x 2048 10.8 / 10.3; 192 rows, 2048 x 7168 15.2 (13.8).  With
// a long K the clusters of 128-row tiles fetch less: 128 rows, 1024 x 16384 15.8 (14.7), 512 x 16384 12.8 (13.5).
// A product whose activations are codes already, which has no quantizer to fetch the first weights under, gains from a K above 1024
// only: 128 rows, 512 x 512 5.6 / 5.0, 1024 x 1024 6.4 / 6.0, 512 x 2048 6.3 / 7.8.
static bool use_rows(int64_t M, int64_t N, int64_t K, bool after_quantizer) {
  const int64_t tiles = ((M + 63) / 64) * ((N + 127) / 128);
  return M <= 64 || (M <= 256 && tiles <= (K <= 8192 ? 32 : 8) && (after_quantizer || K > 1024));
}

uint32_t g_gemm_wait_probes = ptx::kProbeLimit;

template <class Cfg>
static size_t gemm_smem_bytes() {
  return (size_t)Cfg::kTileArea + sizeof(SharedCtl<Cfg>) + 1024;
}

template <Form kForm, int BN>
static int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const CUtensorMap& ma32,
                       const GemmParams& p, int64_t max_units, cudaStream_t st, int sm_margin = 0) {
  const size_t smem = gemm_smem_bytes<TileCfg<BN, kForm>>();
  static thread_local bool attr_set[64] = {false};  // the opt-in is per function and per device
  int dev = 0;
  SGLB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    SGLB_CUDA(cudaFuncSetAttribute(fp8_blockscale_gemm_kernel<kForm, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  int sms = sm_count() - sm_margin;  // SMs left free run a concurrent kernel (the reduce-and-gather of an earlier chunk)
  if (sms < 1) sms = 1;
  const unsigned grid = (unsigned)(max_units < sms ? max_units : sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1), cfg.blockDim = dim3(kGemmThreads, 1, 1), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  if constexpr (kForm == Form::kSplit) {  // (max_units: CTAs, as many as clusters have room at once)
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.splits, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.gridDim.x = (unsigned)max_units, cfg.numAttrs = 2;
    SGLB_CUDA(cudaLaunchKernelEx(&cfg, fp8_blockscale_gemm_kernel<kForm, BN>, ma, mb, mc, ma32, p));
    return SGLB200_OK;
  }
  // A single wave is launched programmatically.  With their quantizer, both ways in turn on one GPU: 100 x 4096 x 4096 15.1 ->
  // 14.4 us, 512 x 4096 x 4096 16.9 -> 16.1, 200 x 8192 x 1024 9.7 -> 9.0; 257 x 10240 x 8192 40.4 -> 39.6, which is less than
  // GPUs and runs differ by.  With several waves the CTAs, which then start wherever an SM falls free, no longer share L2 as
  // their numbers suggest: 4096 x 32768 x 512 114.4 -> 120.9.  Push mode, which other streams take part in: an ordinary launch.
  cfg.numAttrs = max_units <= sms && p.push_maps == nullptr ? 1 : 0;
  SGLB_CUDA(cudaLaunchKernelEx(&cfg, fp8_blockscale_gemm_kernel<kForm, BN>, ma, mb, mc, ma32, p));
  return SGLB200_OK;
}

template <int BN>
static int dense_mm(const DensePlan& dp, const void* A, const void* B, const float* a_s, const float* b_s, void* C,
                    const void* bias, int64_t M, int64_t N, int64_t K, int64_t as_stride_m, int64_t as_stride_k,
                    int out_dtype, void* workspace, int64_t workspace_bytes, bool after_quantizer, cudaStream_t st) {
  CUtensorMap ma, mb;
  int rc = get_tensor_map(A, (uint64_t)K, (uint64_t)M, 1, BM, 2, &ma);
  if (rc) return rc;
  // B is addressed as [1][N][K] so that dense and grouped kernels share the 3-D load
  rc = get_tensor_map(B, (uint64_t)K, (uint64_t)N, 1, BN, 3, &mb);
  if (rc) return rc;
  GemmParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = C, p.bias = bias;
  p.M = M, p.N = N, p.K = K;
  p.as_stride_m = as_stride_m, p.as_stride_k = as_stride_k;
  p.kb_total = (int)((K + BK - 1) / BK), p.nb_total = (int)((N + kScaleBlockN - 1) / kScaleBlockN);
  p.tiles_n = (int)((N + BN - 1) / BN);
  p.group_m = choose_group_m(M, K, BM);
  p.out_fp16 = out_dtype;
  p.wait_probes = g_gemm_wait_probes;
  p.early_weights = after_quantizer ? 1 : 0;
  const int64_t tiles = ((M + BM - 1) / BM) * p.tiles_n;
  if constexpr (BN == 128) {
    if (dp.cluster > 1) {
      p.splits = dp.cluster;
      return launch_gemm<Form::kSplit, BN>(ma, mb, ma, ma, p, tiles * dp.cluster, st);
    }
  }
  UnitPlan pl = dp.units;
  if (pl.scratch_blocks() > 0 &&
      (workspace == nullptr || !aligned16(workspace) || workspace_bytes < dp.scratch_bytes()))
    pl = UnitPlan{(int)tiles, 1, p.kb_total, 0, 0, 0, 2};  // no scratch offered: one unit per tile
  p.full_units = pl.full_units, p.splits = pl.splits, p.kb_per_split = pl.kb_per_split;
  p.sk_share = pl.sk_share, p.sk_ctas = pl.sk_ctas, p.sk_pieces = pl.sk_pieces, p.sk_total = (int)(tiles * p.kb_total);
  p.partial = static_cast<float*>(workspace);
  CUtensorMap mc{};
  p.tma_out = pl.sk_share == 0 && pl.full_units > 0;
  if (p.tma_out) {
    rc = get_out_map(C, (uint64_t)N, (uint64_t)M, out_dtype, BM, &mc);
    if (rc) return rc;
  }
  const int64_t units = pl.sk_share > 0 ? pl.sk_ctas : pl.full_units + pl.split_tiles * pl.splits;
  const bool once = p.kb_total >= (units >= (M <= BM ? 32 : 96) ? 12 : 32) && (!p.tma_out || units <= sm_count());
  rc = once ? launch_gemm<Form::kOnce, BN>(ma, mb, mc, ma, p, units, st) : launch_gemm<Form::kDense, BN>(ma, mb, mc, ma, p, units, st);
  if (rc != SGLB200_OK || pl.scratch_blocks() == 0) return rc;
  const int tiles_m = (int)((M + BM - 1) / BM);
  const unsigned ygrid = (unsigned)((BM * BN / 8 + 255) / 256);
  // The reduction is launched programmatically (it may be scheduled while the GEMM's last CTAs drain).
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int bn = BN;
  if (pl.sk_share > 0) {
    cfg.gridDim = dim3((unsigned)tiles, ygrid, 1);
    if (out_dtype == 0)
      SGLB_CUDA(cudaLaunchKernelEx(&cfg, streamk_reduce_kernel<__nv_bfloat16>, (const float*)p.partial,
                                   static_cast<__nv_bfloat16*>(C), static_cast<const __nv_bfloat16*>(bias), M, N, bn,
                                   tiles_m, p.tiles_n, p.group_m, p.kb_total, pl.sk_share, pl.sk_ctas));
    else
      SGLB_CUDA(cudaLaunchKernelEx(&cfg, streamk_reduce_kernel<__half>, (const float*)p.partial, static_cast<__half*>(C),
                                   static_cast<const __half*>(bias), M, N, bn, tiles_m, p.tiles_n, p.group_m,
                                   p.kb_total, pl.sk_share, pl.sk_ctas));
    return SGLB200_OK;
  }
  cfg.gridDim = dim3((unsigned)pl.split_tiles, ygrid, 1);
  if (out_dtype == 0)
    SGLB_CUDA(cudaLaunchKernelEx(&cfg, split_reduce_kernel<__nv_bfloat16>, (const float*)p.partial,
                                 static_cast<__nv_bfloat16*>(C), static_cast<const __nv_bfloat16*>(bias), M, N, bn, tiles_m,
                                 p.tiles_n, p.group_m, pl.full_units, pl.splits));
  else
    SGLB_CUDA(cudaLaunchKernelEx(&cfg, split_reduce_kernel<__half>, (const float*)p.partial, static_cast<__half*>(C),
                                 static_cast<const __half*>(bias), M, N, bn, tiles_m, p.tiles_n, p.group_m,
                                 pl.full_units, pl.splits));
  return SGLB200_OK;
}

template <int BN>
static int grouped_mm(const void* A, const float* a_s, const void* B, const float* b_s, void* C,
                      const int32_t* sorted_token_ids, const int32_t* expert_ids, const int32_t* num_rows_dev,
                      const float* row_weights, int64_t max_rows, int64_t numel, int num_experts, int64_t N, int64_t K,
                      int scatter, int out_dtype, Padding padding, cudaStream_t st) {
  CUtensorMap ma, mb, ma32;
  int rc = get_tensor_map(A, (uint64_t)K, (uint64_t)max_rows, 1, BM, 2, &ma);
  if (rc) return rc;
  rc = get_tensor_map(A, (uint64_t)K, (uint64_t)max_rows, 1, 32, 2, &ma32);
  if (rc) return rc;
  rc = get_tensor_map(B, (uint64_t)K, (uint64_t)N, (uint64_t)num_experts, BN, 3, &mb);
  if (rc) return rc;
  GemmParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = C, p.bias = nullptr;
  p.sorted_ids = sorted_token_ids, p.expert_ids = expert_ids, p.num_rows_dev = num_rows_dev;
  p.row_weights = scatter || padding != Padding::kKept ? row_weights : nullptr;  // (elsewhere the sorted rows are the bare product, and may have no ids)
  p.M = max_rows, p.N = N, p.K = K;
  p.kb_total = (int)((K + BK - 1) / BK), p.nb_total = (int)((N + kScaleBlockN - 1) / kScaleBlockN);
  p.tiles_n = (int)((N + BN - 1) / BN);
  p.group_m = choose_group_m(max_rows, K, BM);
  p.as_stride_m = p.kb_total, p.as_stride_k = 1;
  p.numel = numel, p.scatter = scatter, p.out_fp16 = out_dtype, p.skip_padding = padding == Padding::kSkipped;
  p.wait_probes = g_gemm_wait_probes;
  p.full_units = 0, p.splits = 1, p.kb_per_split = p.kb_total, p.partial = nullptr;  // grouped: one unit per tile
  p.sk_pieces = 2;
  CUtensorMap mc{};
  p.tma_out = !scatter;  // sorted-row output is contiguous; the scatter form writes token-major rows one by one
  if (p.tma_out) {
    rc = get_out_map(C, (uint64_t)N, (uint64_t)max_rows, out_dtype, p.skip_padding ? 32 : BM, &mc);
    if (rc) return rc;
  }
  const int64_t tiles = ((max_rows + BM - 1) / BM) * p.tiles_n;
  return launch_gemm<Form::kGrouped, BN>(ma, mb, mc, ma32, p, tiles, st);
}

// The first product of the routed experts with the activation and its quantizer in the epilogue (rows as grouped_mm):
// codes [max_rows][I] and scales [max_rows][I / 128] of silu(A w_gate) * (A w_up), w13 = [E][2 I][K].  Quadrants of padding are
// not written.
int grouped_act_mm(const void* A, const float* a_s, const void* w13, const float* b_s, void* out_q, float* out_s,
                   const int32_t* sorted_ids, const int32_t* expert_ids, const int32_t* num_rows_dev, int64_t max_rows,
                   int64_t numel, int num_experts, int64_t I, int64_t K, int dtype, cudaStream_t st) {
  CUtensorMap ma, mb, mc, ma32;
  int rc = get_tensor_map(A, (uint64_t)K, (uint64_t)max_rows, 1, BM, 2, &ma);
  if (rc) return rc;
  rc = get_tensor_map(w13, (uint64_t)K, (uint64_t)(2 * I), (uint64_t)num_experts, 128, 3, &mb);
  if (rc) return rc;
  rc = get_tensor_map(A, (uint64_t)K, (uint64_t)max_rows, 1, 32, 2, &ma32);
  if (rc) return rc;
  rc = get_tensor_map(out_q, (uint64_t)I, (uint64_t)max_rows, 1, 32, 2, &mc);
  if (rc) return rc;
  GemmParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = out_q, p.act_s = out_s;
  p.tma_out = 1;
  p.sorted_ids = sorted_ids, p.expert_ids = expert_ids, p.num_rows_dev = num_rows_dev;
  p.numel = numel, p.skip_padding = 1;
  p.M = max_rows, p.N = 2 * I, p.K = K;
  p.kb_total = (int)(K / BK), p.nb_total = (int)(2 * I / kScaleBlockN);
  p.tiles_n = (int)(I / 128);
  p.group_m = choose_group_m(max_rows, K, BM);
  p.as_stride_m = p.kb_total, p.as_stride_k = 1;
  p.out_fp16 = dtype;
  p.wait_probes = g_gemm_wait_probes;
  p.splits = 1, p.kb_per_split = p.kb_total, p.sk_pieces = 2;
  return launch_gemm<Form::kActivated, 256>(ma, mb, mc, ma32, p, (max_rows + BM - 1) / BM * p.tiles_n, st);
}

}  // namespace sglb200

using namespace sglb200;

extern "C" int sglb200_gemm_status_clear(void) {
  const int zero = 0;
  SGLB_CUDA(cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int)));
  const int rc = rows_gemm_status_clear();
  return rc != SGLB200_OK ? rc : small_linear_status_clear();
}

extern "C" int sglb200_gemm_status(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemm_status, sizeof(int)) != cudaSuccess) return -1;
  if (v == 0) v = rows_gemm_status();
  return v != 0 ? v : small_linear_status();
}

extern "C" void sglb200_gemm_set_wait_probes(uint32_t probes) { g_gemm_wait_probes = probes == 0 ? ptx::kProbeLimit : probes; }

extern "C" int64_t sglb200_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0 || use_rows(M, N, K, true)) return 0;  // (what a plain product of such a size takes needs none)
  return plan_dense(M, N, K).scratch_bytes();
}

extern "C" int sglb200_fp8_blockwise_scaled_mm(const void* A, const void* B, const float* a_s, const float* b_s,
                                               void* C, const void* bias, int64_t M, int64_t N, int64_t K,
                                               int64_t as_stride_m, int64_t as_stride_k, int out_dtype,
                                               void* workspace, int64_t workspace_bytes, void* stream) {
  return scaled_mm(A, B, a_s, b_s, C, bias, M, N, K, as_stride_m, as_stride_k, out_dtype, workspace, workspace_bytes, false,
                   static_cast<cudaStream_t>(stream));
}

int sglb200::scaled_mm(const void* A, const void* B, const float* a_s, const float* b_s, void* C, const void* bias, int64_t M,
                       int64_t N, int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype, void* workspace,
                       int64_t workspace_bytes, bool after_quantizer, cudaStream_t st) {
  SGLB_REQUIRE(M >= 0 && N > 0 && K > 0, "fp8_blockwise_scaled_mm: bad shape M=%lld N=%lld K=%lld", (long long)M,
               (long long)N, (long long)K);
  SGLB_REQUIRE(K % 16 == 0, "fp8_blockwise_scaled_mm: K=%lld must be a multiple of 16", (long long)K);
  SGLB_REQUIRE(N % 8 == 0, "fp8_blockwise_scaled_mm: N=%lld must be a multiple of 8", (long long)N);
  SGLB_REQUIRE(out_dtype == 0 || out_dtype == 1, "fp8_blockwise_scaled_mm: out_dtype %d (0 bf16, 1 fp16)", out_dtype);
  if (M == 0) return SGLB200_OK;
  SGLB_REQUIRE(A && B && a_s && b_s && C, "fp8_blockwise_scaled_mm: null pointer");
  SGLB_REQUIRE(aligned16(A) && aligned16(B) && aligned16(C) && (bias == nullptr || aligned16(bias)),
               "fp8_blockwise_scaled_mm: A, B, C and bias must be 16-byte aligned");
  SGLB_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "fp8_blockwise_scaled_mm: dimension too large");
  if (use_rows(M, N, K, after_quantizer))
    return rows_dense_mm(A, B, a_s, b_s, C, bias, M, N, K, as_stride_m, as_stride_k, out_dtype, after_quantizer, st);
  const DensePlan dp = plan_dense(M, N, K);
  if (dp.bn == 128)
    return dense_mm<128>(dp, A, B, a_s, b_s, C, bias, M, N, K, as_stride_m, as_stride_k, out_dtype, workspace,
                         workspace_bytes, after_quantizer, st);
  return dense_mm<256>(dp, A, B, a_s, b_s, C, bias, M, N, K, as_stride_m, as_stride_k, out_dtype, workspace,
                       workspace_bytes, after_quantizer, st);
}

extern "C" int sglb200_fp8_blockwise_grouped_mm(const void* A, const float* a_s, const void* B, const float* b_s,
                                                void* C, const int32_t* sorted_token_ids, const int32_t* expert_ids,
                                                const int32_t* num_rows_dev, const float* row_weights,
                                                int64_t max_rows, int64_t numel, int num_experts, int64_t N, int64_t K,
                                                int scatter, int out_dtype, void* stream) {
  return sglb200::grouped_mm_any(A, a_s, B, b_s, C, sorted_token_ids, expert_ids, num_rows_dev, row_weights, max_rows, numel,
                                 num_experts, N, K, scatter, out_dtype, Padding::kKept, static_cast<cudaStream_t>(stream));
}

int sglb200::grouped_mm_any(const void* A, const float* a_s, const void* B, const float* b_s, void* C,
                            const int32_t* sorted_token_ids, const int32_t* expert_ids, const int32_t* num_rows_dev,
                            const float* row_weights, int64_t max_rows, int64_t numel, int num_experts, int64_t N, int64_t K,
                            int scatter, int out_dtype, Padding padding, cudaStream_t st) {
  SGLB_REQUIRE(max_rows >= 0 && N > 0 && K > 0 && num_experts >= 1, "grouped_mm: bad shape rows=%lld N=%lld K=%lld E=%d",
               (long long)max_rows, (long long)N, (long long)K, num_experts);
  SGLB_REQUIRE(K % 16 == 0 && N % 8 == 0, "grouped_mm: K must be a multiple of 16 and N of 8");
  SGLB_REQUIRE(out_dtype == 0 || out_dtype == 1, "grouped_mm: out_dtype %d (0 bf16, 1 fp16)", out_dtype);
  if (max_rows == 0) return SGLB200_OK;
  SGLB_REQUIRE(A && a_s && B && b_s && C && expert_ids && num_rows_dev, "grouped_mm: null pointer");
  SGLB_REQUIRE((!scatter && padding == Padding::kKept) || sorted_token_ids, "grouped_mm: scatter mode needs sorted_token_ids");
  SGLB_REQUIRE(aligned16(A) && aligned16(B) && aligned16(C), "grouped_mm: A, B and C must be 16-byte aligned");
  if (choose_bn_grouped(numel) == 128)
    return grouped_mm<128>(A, a_s, B, b_s, C, sorted_token_ids, expert_ids, num_rows_dev, row_weights, max_rows, numel,
                           num_experts, N, K, scatter, out_dtype, padding, st);
  return grouped_mm<256>(A, a_s, B, b_s, C, sorted_token_ids, expert_ids, num_rows_dev, row_weights, max_rows, numel,
                         num_experts, N, K, scatter, out_dtype, padding, st);
}


// ---------------------------------------------------------------------------------------------
// Push mode: the GEMM of a row-parallel layer with the reduce-scatter folded into its epilogue.
// ---------------------------------------------------------------------------------------------
namespace sglb200 {

// Device copy of the per-owner output tensor maps, built once per (staging buffers, shape) and kept.
struct PushKey {
  const void* ptrs[8];
  uint64_t N, rows;
  int world, out_fp16;
  bool operator==(const PushKey& o) const {
    for (int i = 0; i < 8; ++i)
      if (ptrs[i] != o.ptrs[i]) return false;
    return N == o.N && rows == o.rows && world == o.world && out_fp16 == o.out_fp16;
  }
};
struct PushKeyHash {
  size_t operator()(const PushKey& k) const {
    size_t h = k.N * 1000003u ^ k.rows;
    for (int i = 0; i < 8; ++i) h = h * 1000003u ^ reinterpret_cast<size_t>(k.ptrs[i]);
    return h * 31u + (size_t)k.world * 2 + (size_t)k.out_fp16;
  }
};

static int get_push_maps(void* const* stage_ptrs, int world, uint64_t N, uint64_t rows, int out_fp16,
                         const CUtensorMap** out) {
  static thread_local std::unordered_map<PushKey, CUtensorMap*, PushKeyHash> cache;
  PushKey key{};
  for (int i = 0; i < world; ++i) key.ptrs[i] = stage_ptrs[i];
  key.N = N, key.rows = rows, key.world = world, key.out_fp16 = out_fp16;
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return SGLB200_OK;
  }
  CUtensorMap host[8];
  for (int i = 0; i < world; ++i) {
    const int rc = get_out_map(stage_ptrs[i], N, rows, out_fp16, BM, &host[i]);
    if (rc) return rc;
  }
  CUtensorMap* dev = nullptr;
  SGLB_CUDA(cudaMalloc(&dev, sizeof(CUtensorMap) * 8));
  SGLB_CUDA(cudaMemcpy(dev, host, sizeof(CUtensorMap) * world, cudaMemcpyHostToDevice));
  cache.emplace(key, dev);
  *out = dev;
  return SGLB200_OK;
}

template <int BN>
static int push_mm(const void* A, const void* B, const float* a_s, const float* b_s, void* const* stage_ptrs, int world,
                   int rank, int64_t M, int64_t N, int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype,
                   int sm_margin, cudaStream_t st) {
  CUtensorMap ma, mb;
  int rc = get_tensor_map(A, (uint64_t)K, (uint64_t)M, 1, BM, 2, &ma);
  if (rc) return rc;
  rc = get_tensor_map(B, (uint64_t)K, (uint64_t)N, 1, BN, 3, &mb);
  if (rc) return rc;
  GemmParams p{};
  p.a_s = a_s, p.b_s = b_s, p.C = nullptr, p.bias = nullptr;
  p.M = M, p.N = N, p.K = K;
  p.as_stride_m = as_stride_m, p.as_stride_k = as_stride_k;
  p.kb_total = (int)((K + BK - 1) / BK), p.nb_total = (int)((N + kScaleBlockN - 1) / kScaleBlockN);
  p.tiles_n = (int)((N + BN - 1) / BN);
  p.group_m = choose_group_m(M, K, BM);
  p.out_fp16 = out_dtype;
  p.wait_probes = g_gemm_wait_probes;
  const int64_t tiles = ((M + BM - 1) / BM) * p.tiles_n;
  p.full_units = (int)tiles, p.splits = 1, p.kb_per_split = p.kb_total, p.partial = nullptr;  // one unit per tile
  p.sk_pieces = 2;
  p.tma_out = 1;
  // rows are owned in blocks of rpo = ceil(M / world) rounded up to whole tiles (the last owners may hold fewer
  // rows, or none); every owner's staging buffer is [world][rpo][N]
  const int64_t rpo = sglb200_push_rows_per_owner(M, world);
  rc = get_push_maps(stage_ptrs, world, (uint64_t)N, (uint64_t)(rpo * world), out_dtype, &p.push_maps);
  if (rc) return rc;
  p.push_rows_per_owner = (int)rpo, p.push_rank = rank;
  CUtensorMap mc = {};
  rc = get_out_map(stage_ptrs[rank], (uint64_t)N, (uint64_t)(rpo * world), out_dtype, BM, &mc);  // unused by the stores; keeps map_c valid
  if (rc) return rc;
  return launch_gemm<Form::kDense, BN>(ma, mb, mc, ma, p, tiles, st, sm_margin);
}

}  // namespace sglb200

extern "C" int64_t sglb200_push_rows_per_owner(int64_t M, int world) {
  if (M <= 0 || world <= 0) return 0;
  const int64_t per = (M + world - 1) / world;
  return (per + BM - 1) / BM * BM;
}

extern "C" int sglb200_push_prepare(void* const* stage_ptrs, int world, int64_t M, int64_t N, int out_dtype) {
  SGLB_REQUIRE(world >= 2 && world <= 8 && stage_ptrs != nullptr, "push_prepare: world %d", world);
  SGLB_REQUIRE(M > 0 && N > 0 && N % 8 == 0 && (out_dtype == 0 || out_dtype == 1), "push_prepare: bad shape or dtype");
  for (int i = 0; i < world; ++i)
    SGLB_REQUIRE(stage_ptrs[i] != nullptr && aligned16(stage_ptrs[i]), "push_prepare: staging buffer %d missing or unaligned", i);
  const int64_t rpo = sglb200_push_rows_per_owner(M, world);
  const CUtensorMap* maps = nullptr;
  return get_push_maps(stage_ptrs, world, (uint64_t)N, (uint64_t)(rpo * world), out_dtype, &maps);
}

extern "C" int sglb200_fp8_blockwise_scaled_mm_push(const void* A, const void* B, const float* a_s, const float* b_s,
                                                    void* const* stage_ptrs, int world, int rank, int64_t M, int64_t N,
                                                    int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype,
                                                    int sm_margin, void* stream) {
  SGLB_REQUIRE(world >= 2 && world <= 8 && rank >= 0 && rank < world, "mm_push: world %d, rank %d", world, rank);
  SGLB_REQUIRE(sm_margin >= 0 && sm_margin < sm_count(), "mm_push: sm_margin %d", sm_margin);
  SGLB_REQUIRE(M > 0 && N > 0 && K > 0, "mm_push: bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N,
               (long long)K);
  SGLB_REQUIRE(K % 16 == 0 && N % 8 == 0, "mm_push: K=%lld must be a multiple of 16 and N=%lld of 8", (long long)K,
               (long long)N);
  SGLB_REQUIRE(out_dtype == 0 || out_dtype == 1, "mm_push: out_dtype %d (0 bf16, 1 fp16)", out_dtype);
  SGLB_REQUIRE(A && B && a_s && b_s && stage_ptrs, "mm_push: null pointer");
  for (int i = 0; i < world; ++i)
    SGLB_REQUIRE(stage_ptrs[i] != nullptr && aligned16(stage_ptrs[i]), "mm_push: staging buffer %d missing or unaligned", i);
  SGLB_REQUIRE(aligned16(A) && aligned16(B), "mm_push: A and B must be 16-byte aligned");
  SGLB_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "mm_push: dimension too large");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (choose_bn(M, N, K, sm_count() - sm_margin) == 128)
    return push_mm<128>(A, B, a_s, b_s, stage_ptrs, world, rank, M, N, K, as_stride_m, as_stride_k, out_dtype, sm_margin, st);
  return push_mm<256>(A, B, a_s, b_s, stage_ptrs, world, rank, M, N, K, as_stride_m, as_stride_k, out_dtype, sm_margin, st);
}

#ifdef SGLB_TRACE
extern "C" int sglb200_debug_trace(void* host_buf, int64_t bytes) {
  if (bytes != (int64_t)sizeof(long long) * 2 * kTraceUnits * kTraceStamps) return -1;
  return cudaMemcpyFromSymbol(host_buf, g_trace, (size_t)bytes) == cudaSuccess ? 0 : -2;
}
#endif
