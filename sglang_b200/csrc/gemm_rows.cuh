// Shared by the kernels with the weights on the M side (gemm_rows.cu, gemm_small.cu): launch parameters, the walk over
// tiles, the count of the experts' token tiles, the sum over the CTAs of a cluster.
#pragma once
#include "cluster_rule.h"
#include "common.cuh"
#include "gemm_common.cuh"
#include "ptx_sm100.cuh"

namespace sglb200 {

constexpr int kRowsBM = 128;                     // weight rows per tile
constexpr int kRowsBK = 128;                     // K slab: one scale block
constexpr uint32_t kWBytes = kRowsBM * kRowsBK;  // weight bytes per stage
constexpr int kScBatch = 8;                      // slabs whose scales are prepared together
constexpr int kMaxExperts = 1024;
constexpr int kMaxSplits = kMostClusterCtas;     // CTAs of a cluster
constexpr int kPartPitch = kRowsBM + 4;          // floats between the columns of a CTA's partial sums
constexpr int kPartPair = 2 * kRowsBM + 8;       // the same between pairs of columns in the pushed form

// Where the scale of column j of a tile lies, so that one 16-byte read gives a thread those of the four columns that it
// holds of 16 (2 c, 2 c + 1, 2 c + 8, 2 c + 9 with c = lane % 4, see ptx::tmem_ld_16x256).
__device__ __forceinline__ int frag_column(int j) { return (j & ~15) + ((j & 7) >> 1) * 4 + ((j >> 3) & 1) * 2 + (j & 1); }
// Tensor memory: a CTA of these kernels takes 128 or 256 of an SM's 512 columns and may find CTAs of the kernel in front
// of it or behind it there, of which the latter wait for this one.  No allocation can wait for them in turn, as an SM that has
// registers for a set of such CTAs has columns for it too: a CTA with 256 columns has 256 threads of at least 110 registers
// (43 % of the file), one with 128 columns 256 threads of at least 74 (31 %) or 288 of 96 (42 %), so that beside one
// with 256 columns there is room for one other of either kind, without one for three of 128.  The 128-row kernel, which takes
// all columns, leaves no registers for another CTA.

struct RowsParams {
  const float* a_s;
  const float* b_s;
  void* C;
  const void* bias;                // dense, optional
  int64_t M, N;                    // dense: rows of A
  int64_t as_stride_m, as_stride_k;
  int kb_total, nb_total, tiles_n;
  int tiles_m;                     // dense
  int splits;                      // CTAs of a cluster, each with its part of K (1 = no cluster)
  uint32_t per_row;                // one-launch linear: g / M = g * per_row >> 16 for the groups of a CTA (g < 128, M <= 16)
  int early_weights;               // the weights may be read before the predecessor in the stream has finished
  int out_fp16;
  int group_m;                     // token tiles of a group sweep over the weight tiles together
  // expert-grouped form
  int num_experts;
  const int32_t* cumsum;           // [experts + 2] padded starts of the buckets (bucket e + 1 = expert e), multiples of 16
  const int32_t* sorted_ids;       // flat top-k slots in expert order, >= numel = padding
  int64_t numel;
  int gather_topk;                 // > 0: A has a row per token, fetched by slot / gather_topk; 0: A is in expert order
  int scatter;                     // write row sorted_ids[r] instead of row r
  const float* row_weights;        // scatter, optional
  int32_t* next_tile;              // a zero: tiles beyond the first of every CTA are taken from this counter; nullptr: in turn
  uint32_t wait_probes;
};

struct alignas(16) RowsTile {
  int n_tile, row0, n_eff, expert;
};

template <int NT, bool kGrouped>
__device__ __forceinline__ RowsTile rows_tile(const RowsParams& p, const int* tiles_before, int t) {
  RowsTile x;
  int m_tile;
  if constexpr (kGrouped) {
    int lo = 0, hi = p.num_experts;  // the expert with tiles_before[e] * tiles_n <= t < tiles_before[e + 1] * tiles_n
    const int tt = t / p.tiles_n;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tiles_before[mid] <= tt) lo = mid; else hi = mid;
    }
    x.expert = lo;
    const int first = tiles_before[lo];
    tile_coord(t - first * p.tiles_n, tiles_before[lo + 1] - first, p.tiles_n, p.group_m, m_tile, x.n_tile);
    const int begin = p.cumsum[lo + 1], end = p.cumsum[lo + 2];
    x.row0 = begin + m_tile * NT;
    x.n_eff = min(NT, end - x.row0);
  } else {
    tile_coord(t, p.tiles_m, p.tiles_n, p.group_m, m_tile, x.n_tile);
    x.expert = 0;
    x.row0 = m_tile * NT;
    x.n_eff = min(NT, ((int)p.M - x.row0 + 15) & ~15);
  }
  return x;
}

// Token tiles (of NT rows) of every expert and their exclusive scan into tiles_before[0 .. experts]: four experts per thread,
// all NTHREADS threads of the block.  The scan is visible after the next __syncthreads.  An expert's first row is read from
// p.cumsum where a tile is located: in shared memory beside the scan, it cost a layer of 128 experts 0.6 us.
template <int NT, int NTHREADS>
__device__ __forceinline__ void rows_count_tiles(const RowsParams& p, int* tiles_before, int* warp_sum) {
  static_assert(NTHREADS * 4 >= kMaxExperts, "four experts per thread");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int cnt[4], mine = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = tid * 4 + k;
    cnt[k] = e < p.num_experts ? (p.cumsum[e + 2] - p.cumsum[e + 1] + NT - 1) / NT : 0;
    mine += cnt[k];
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int before = incl - mine;
  for (int w = 0; w < warp; ++w) before += warp_sum[w];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = tid * 4 + k;
    if (e < p.num_experts) tiles_before[e] = before;
    before += cnt[k];
  }
  if (tid == NTHREADS - 1) tiles_before[p.num_experts] = before;  // (experts beyond num_experts count 0)
}

// The output of a tile whose K range was split over the CTAs of a cluster (at most kMost): sums their partial sums
// ([column][kPartPitch weight rows] of float32 at `part` in every CTA's shared memory) in ascending K order, adds the bias,
// rounds once.
template <int kMost>
__device__ __forceinline__ void rows_cluster_sum(const RowsParams& p, const RowsTile& x, int rank, uint32_t part, int tid,
                                                 int threads) {
  const int splits = p.splits;
  // CTA `rank` adds columns rank, rank + splits, ..; a thread adds two neighbouring weight rows of a column
  const int mine = (x.n_eff - rank + splits - 1) / splits;
  for (int i = tid; i < mine * (kRowsBM / 2); i += threads) {
    const int col = rank + (i / (kRowsBM / 2)) * splits, pair = i % (kRowsBM / 2);
    const int n = x.n_tile * kRowsBM + pair * 2, row = x.row0 + col;
    if (n >= p.N || row >= p.M) continue;
    float2 v[kMost];
#pragma unroll
    for (int s = 0; s < kMost; ++s)  // all requested before the first is added
      if (s < splits) v[s] = ptx::lds_cluster_f32x2(ptx::cluster_map(part + (col * kPartPitch + pair * 2) * 4, s));
    float a = v[0].x, b = v[0].y;
#pragma unroll
    for (int s = 1; s < kMost; ++s)
      if (s < splits) a += v[s].x, b += v[s].y;
    uint32_t word;
    if (p.out_fp16) {
      if (p.bias != nullptr) {
        const __half* bs = static_cast<const __half*>(p.bias) + n;
        a += __half2float(bs[0]), b += __half2float(bs[1]);
      }
      const __half2 o = __floats2half2_rn(a, b);
      word = *reinterpret_cast<const uint32_t*>(&o);
    } else {
      if (p.bias != nullptr) {
        const __nv_bfloat16* bs = static_cast<const __nv_bfloat16*>(p.bias) + n;
        a += __bfloat162float(bs[0]), b += __bfloat162float(bs[1]);
      }
      const __nv_bfloat162 o = __floats2bfloat162_rn(a, b);
      word = *reinterpret_cast<const uint32_t*>(&o);
    }
    *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(p.C) + (int64_t)row * p.N + n) = word;
  }
}

// The same for tiles of 64 columns, pushed instead of fetched: a CTA owns the pairs of neighbouring columns rank, rank +
// splits, .., every CTA writes the others' partial sums straight into their shared memory ([source CTA][owned pair][2][128
// rows] at `part`), and after a barrier all that is left is local.  Fetched (written, barrier, read across the cluster, barrier
// before anyone may leave) the exchange takes 3.4 of the kernel's 8.6 us of 64 x 4096 x 4096; the layer with its quantizer
// 10.9 us so and 10.1 pushed, 512 x 512 7.2 and 6.4, 4096 x 14336 17.5 and 16.2.  With 16 or 32 columns there is little
// to exchange and the barrier before the first remote write costs more than that saves (32 x 1024 x 8192 7.6 and 8.0).
//
// Every thread of the cluster arrives and waits twice: the first time when its CTA's operands, which `part` lies over, have
// been consumed, the second time when its partial sums are written.
__device__ __forceinline__ int cluster_pairs(const RowsTile& x, int splits) { return (x.n_eff / 2 + splits - 1) / splits; }

// One thread's part of `kUnits` times eight columns from `col0` on: acc[half][4 u ..] as tmem_ld_16x256 has them, of quadrant q.
template <int kUnits>
__device__ __forceinline__ void rows_cluster_put(const RowsParams& p, const RowsTile& x, int rank, uint32_t part, const float* acc0,
                                                 const float* acc1, int col0, int q, int lane) {
  const int splits = p.splits, pairs = cluster_pairs(x, splits), rows = min(x.n_eff, (int)p.M - x.row0);
  const uint32_t mine = part + (uint32_t)(rank * pairs * kPartPair + q * 32 + (lane >> 2) * 4) * 4;
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const int pair = col0 / 2 + 4 * u + (lane & 3);
    if (2 * pair < rows) {
      const int idx = pair / splits;
      const uint32_t to = ptx::cluster_map(mine + (uint32_t)(idx * kPartPair) * 4, pair - idx * splits);
      ptx::sts_cluster_f32x4(to, acc0[4 * u], acc0[4 * u + 2], acc1[4 * u], acc1[4 * u + 2]);
      ptx::sts_cluster_f32x4(to + kRowsBM * 4, acc0[4 * u + 1], acc0[4 * u + 3], acc1[4 * u + 1], acc1[4 * u + 3]);
    }
  }
}

// The owned columns: partial sums in ascending K order, bias, one rounding.  A warp takes 32 weight rows of four pairs.
__device__ __forceinline__ void rows_cluster_get(const RowsParams& p, const RowsTile& x, int rank, uint32_t part, int warp, int warps,
                                                 int lane) {
  const int splits = p.splits, pairs = cluster_pairs(x, splits);
  for (int t = warp; t < 4 * ((pairs + 3) / 4); t += warps) {  // (uniform over the warp)
    const int q = t & 3, first = (t >> 2) * 4, idx = first + (lane & 3);
    float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
    if (idx < pairs && 2 * (rank + splits * idx) < (int)p.M - x.row0) {  // (pairs past the last row are not written)
      uint32_t from = part + (uint32_t)(idx * kPartPair + q * 32 + (lane >> 2) * 4) * 4;
#pragma unroll 4
      for (int s = 0; s < splits; ++s, from += (uint32_t)(pairs * kPartPair) * 4) {
        const float4 v = ptx::lds_f32x4(from), w = ptx::lds_f32x4(from + kRowsBM * 4);
        a[0] += v.x, a[1] += v.y, a[2] += v.z, a[3] += v.w;
        b[0] += w.x, b[1] += w.y, b[2] += w.z, b[3] += w.w;
      }
    }
    const int n0 = x.n_tile * kRowsBM + q * 32;
    uint32_t m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float bias = 0.f;
      const int n = min(n0 + 8 * k + (lane >> 2), (int)p.N - 1);
      if (p.out_fp16) {
        if (p.bias != nullptr) bias = __half2float(static_cast<const __half*>(p.bias)[n]);
        const __half2 o = __floats2half2_rn(a[k] + bias, b[k] + bias);
        m[k] = *reinterpret_cast<const uint32_t*>(&o);
      } else {
        if (p.bias != nullptr) bias = __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[n]);
        const __nv_bfloat162 o = __floats2bfloat162_rn(a[k] + bias, b[k] + bias);
        m[k] = *reinterpret_cast<const uint32_t*>(&o);
      }
    }
    const uint4 v = ptx::transpose_frags(m, lane);
    const int c = lane >> 2, mine = first + (c >> 1), col = 2 * (rank + splits * mine) + (c & 1), row = x.row0 + col;
    const int n = n0 + (lane & 3) * 8;  // (N is a multiple of 8)
    if (mine < pairs && col < x.n_eff && row < p.M && n < p.N)
      *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.C) + (int64_t)row * p.N + n) = v;
  }
}

#define ROWS_WAIT(bar, parity) \
  (p.wait_probes != ptx::kProbesNone && (ptx::mbar_test(bar, parity) || ptx::mbar_wait_quiet(bar, parity)))

}  // namespace sglb200
