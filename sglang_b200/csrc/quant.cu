// 1 x G activation quantizer (float8_e4m3fn codes + float32 scales) and the fused
// silu_and_mul + quantizer, for sm_100a.
//
// Both are bound by HBM, and have two forms.  Direct: a thread loads 16 elements of one group straight into registers
// (one 256-bit load for 16-bit types), the group maximum takes log2(G / 16) shuffles, and the 16 codes leave in one
// 128-bit store; no shared memory and no barrier, so no warp waits for another.  Ring (large 16-bit inputs of the quantizer,
// masked expert batches of the activation): persistent CTAs walk tiles of 8192 elements that one thread stages with bulk
// copies (cp.async.bulk) into a ring of shared-memory buffers completing on mbarriers, so the bytes in flight per SM do
// not depend on registers or occupancy; a thread owns 32 elements of one group per tile.
//
// Arithmetic contract (bit-exact with the reference CUDA kernel built without fast-math):
//   amax  = max(|x|, eps)            scale = amax / fp8_max      (div.rn.f32)
//   code  = cvt.rn.satfinite.e4m3( min(max(x / scale, fp8_min), fp8_max) )   (div.rn.f32)
#include "common.cuh"
#include "gemm_common.cuh"
#include "ptx_sm100.cuh"
#include "quant_math.cuh"

namespace sglb200 {

// ---- ring: streaming skeleton shared by the quantizer and the masked activation + quantizer --------------
//
// A CTA walks tiles of kTileElems consecutive elements (tile t, t + gridDim.x, ...).  One thread stages
// each tile with a 1-D bulk copy (cp.async.bulk) into a ring of kStreamStages shared-memory buffers that
// complete on mbarriers, so the bytes in flight per SM are set by the ring and not by registers or
// occupancy.  A thread owns kThreadElems = 32 elements of ONE group per tile (a 128-group is shared by four
// lanes: two shuffle rounds per 32 elements), read as 16-byte chunks interleaved over the lanes of the
// group so that shared-memory reads are conflict-free and every quad of lanes writes one full 32-byte
// sector of codes.
constexpr int kStreamThreads = 256;
constexpr int kTileElems = kStreamThreads * kThreadElems;  // 8192
template <typename T>
constexpr int kStagesOf = sizeof(T) == 4 ? 3 : 4;  // 64 KB (16-bit types) or 96 KB (float32) of ring per CTA

__device__ int g_stream_status = 0;  // 0 ok, 1 = a wait for a staged tile expired
static uint32_t g_stream_wait_probes = ptx::kProbeLimit;  // sglb200_stream_set_wait_probes

// A CTA that gave up a wait: it records the failure and then holds its shared memory for about a millisecond, so
// that bulk copies it has already issued into other ring slots land before the SM hands the memory to another CTA.
__device__ __forceinline__ void stream_give_up(int tid) {
  if (tid == 0) {
    atomicExch(&g_stream_status, 1);
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Interleaving of a group's 16-byte chunks over its LPG lanes: lane l reads chunk (LPG * j + l + rot) mod GC at
// step j, where rot depends on the group's position so that the eight threads of a quarter warp always touch
// eight different 16-byte bank groups.
template <typename T, int LPG>
__device__ __forceinline__ int chunk_rotation(int g) {
  constexpr int GC = LPG * Chunk<T>::kPerThread;  // chunks per group
  if (LPG >= 8) return 0;
  if (LPG == 1) return GC >= 8 ? (g & 7) : ((g >> 1) & (GC - 1));
  return LPG * (g & (8 / LPG - 1));
}

// The quantizer.  `issue(i)` (thread 0) arms the slot's mbarrier with the byte count of this CTA's i-th tile and
// starts its copy.

template <typename T, int LPG, bool kStdRange>
__global__ void __launch_bounds__(kStreamThreads, 3)
    quant_stream_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q, float* __restrict__ out_s,
                        int64_t total_elems, int groups_per_row, int64_t s_stride_token, int64_t s_stride_group,
                        bool s_contiguous, float eps, float qmin, float qmax, uint32_t probes, bool trigger) {
  constexpr int CE = Chunk<T>::kElems, NCH = Chunk<T>::kPerThread, GC = LPG * NCH;
  constexpr int G = LPG * kThreadElems;
  constexpr int kStreamStages = kStagesOf<T>;
  constexpr uint32_t kTileBytes = kTileElems * sizeof(T);
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kStreamStages];
  __shared__ int s_abort;
  const uint32_t smem_base = ptx::smem_u32(smem_raw);
  const int tid = threadIdx.x;
  const int64_t tiles = (total_elems + kTileElems - 1) / kTileElems;
  const int64_t my_tiles = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;  // > 0: the grid never exceeds tiles

  auto issue = [&](int64_t i) {  // thread 0 only
    const int slot = (int)(i % kStreamStages);
    const int64_t e0 = (blockIdx.x + i * gridDim.x) * (int64_t)kTileElems;
    const int64_t left = total_elems - e0;
    const uint32_t bytes = left >= kTileElems ? kTileBytes : (uint32_t)(left * sizeof(T));
    const uint32_t bar = ptx::smem_u32(&bars[slot]);
    ptx::mbar_arrive_expect_tx(bar, bytes);
    bulk_load_1d(smem_base + slot * kTileBytes, x + e0, bytes, bar);
  };

  if (tid == 0) {
    s_abort = 0;
#pragma unroll
    for (int s = 0; s < kStreamStages; ++s) ptx::mbar_init(ptx::smem_u32(&bars[s]), 1);
    ptx::mbar_fence_init();
  }
  // In this order: what is launched on the trigger may then count on everything before this kernel being complete and
  // visible (the rows kernel of the same linear layer reads its weights at once).  Only a call whose next launch is its own
  // triggers; what follows a kernel that writes for the caller starts when that is done.
  ptx::grid_dependency_wait();
  if (trigger) ptx::launch_dependents();
  if (tid == 0) {
    for (int64_t i = 0; i < kStreamStages && i < my_tiles; ++i) issue(i);
  }
  __syncthreads();

  const int g_local = tid / LPG, l = tid % LPG;
  const int rot = chunk_rotation<T, LPG>(g_local);
  int cj[NCH];
#pragma unroll
  for (int j = 0; j < NCH; ++j) cj[j] = (LPG * j + l + rot) % GC;

  for (int64_t i = 0; i < my_tiles; ++i) {
    const int slot = (int)(i % kStreamStages);
    const uint32_t parity = (uint32_t)((i / kStreamStages) & 1);
    if (!ptx::mbar_probe(ptx::smem_u32(&bars[slot]), parity, probes)) s_abort = 1;
    uint4 raw[NCH];
    const uint32_t src = smem_base + slot * kTileBytes + (uint32_t)(g_local * GC) * 16u;
#pragma unroll
    for (int j = 0; j < NCH; ++j) raw[j] = ptx::lds_128(src + (uint32_t)cj[j] * 16u);
    __syncthreads();  // every thread holds its part of the slot in registers: the slot can be refilled
    if (s_abort) {  // (uniform: read after the barrier)
      stream_give_up(tid);
      return;
    }
    if (tid == 0 && i + kStreamStages < my_tiles) issue(i + kStreamStages);

    float v[NCH * CE];
#pragma unroll
    for (int j = 0; j < NCH; ++j) unpack_chunk<T>(raw[j], v + j * CE);
    uint32_t codes[NCH][CE / 4];
    const float scale = quant_group<T, LPG, kStdRange>(raw, v, eps, qmin, qmax, codes);

    const int64_t e0 = (blockIdx.x + i * gridDim.x) * (int64_t)kTileElems;
    const int64_t ge = e0 + (int64_t)g_local * G;  // first element of this thread's group
    if (ge < total_elems) {
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        uint8_t* dst = out_q + ge + cj[j] * CE;
        if constexpr (CE == 8) {
          *reinterpret_cast<uint2*>(dst) = make_uint2(codes[j][0], codes[j][1]);
        } else {
          *reinterpret_cast<uint32_t*>(dst) = codes[j][0];
        }
      }
      if (l == 0) {
        const int64_t g = ge / G;
        if (s_contiguous) {
          out_s[g] = scale;
        } else {
          const int64_t t = g / groups_per_row;
          out_s[t * s_stride_token + (g - t * groups_per_row) * s_stride_group] = scale;
        }
      }
    }
  }
}

// ---- direct forms: values straight to registers ---------------------------------------------------------

constexpr int kQuantThreads = 256;
constexpr int kLaneElems = 16;                            // elements of one group that a thread owns
constexpr int kUnitElems = kQuantThreads * kLaneElems;    // 4096

// A thread's 16 elements: `wide` (32-byte aligned) in 256-bit loads, else in 128-bit ones.
template <int N>
__device__ __forceinline__ void load_lane(uint4* r, const void* p, bool wide) {
  const uint8_t* b = static_cast<const uint8_t*>(p);
  if (wide) {
#pragma unroll
    for (int j = 0; j < N; j += 2)
      asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(r[j].x), "=r"(r[j].y), "=r"(r[j].z), "=r"(r[j].w), "=r"(r[j + 1].x), "=r"(r[j + 1].y),
                     "=r"(r[j + 1].z), "=r"(r[j + 1].w)
                   : "l"(b + j * 16));
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j)
      asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(r[j].x), "=r"(r[j].y), "=r"(r[j].z), "=r"(r[j].w)
                   : "l"(b + j * 16));
  }
}
__device__ __forceinline__ void store_lane(uint8_t* p, const uint32_t* c, bool wide) {
  if (wide) {
    *reinterpret_cast<uint4*>(p) = make_uint4(c[0], c[1], c[2], c[3]);
  } else {
    reinterpret_cast<uint2*>(p)[0] = make_uint2(c[0], c[1]);
    reinterpret_cast<uint2*>(p)[1] = make_uint2(c[2], c[3]);
  }
}
// Quotient of a group index; almost always both fit 32 bits, and a 64-bit division is a function call.
__device__ __forceinline__ int64_t div_groups(int64_t g, int per_row) {
  return g < (1ll << 32) ? (int64_t)((uint32_t)g / (uint32_t)per_row) : g / per_row;
}

struct ScaleLayout {
  int groups_per_row;
  int64_t stride_token, stride_group;
  bool contiguous;  // [token][group], dense
};

// The quantizer, direct form.  A thread has U units of 16 elements in flight.
// kTiled: for scales with adjacent tokens in adjacent words (the GEMM's layout).  The flat order writes them one word
// per sector; here a warp takes one group column and its groups are 32 / LPG adjacent tokens in each unit, so that one
// store instruction writes U * 32 / LPG adjacent scales - for groups of 128 exactly one sector - while the eight warps
// of a CTA still read 2 KB runs of every row.
template <typename T, int LPG, bool kStdRange, int U, bool kTiled>
__global__ void __launch_bounds__(kQuantThreads)
    quant_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q, float* __restrict__ out_s, int64_t tokens,
                 ScaleLayout sl, float eps, float qmin, float qmax, bool wide_in, bool wide_out, bool trigger) {
  constexpr int CE = Chunk<T>::kElems, NCH = kLaneElems / CE, G = LPG * kLaneElems;
  constexpr int kWarpGroups = 32 / LPG;
  static_assert(U <= LPG, "one lane of the group stores each unit's scale");
  // In this order: what is launched on the trigger may then count on everything before this kernel being complete and
  // visible (the rows kernel of the same linear layer reads its weights at once).  Only a call whose next launch is its own
  // triggers; what follows a kernel that writes for the caller starts when that is done.
  ptx::grid_dependency_wait();
  if (trigger) ptx::launch_dependents();
  const int l = threadIdx.x % LPG, slot = (threadIdx.x & 31) / LPG, warp = threadIdx.x >> 5;
  int64_t ge[U];  // first element of the thread's group in each unit, -1 beyond the end
  int64_t row0 = 0;
  int col = 0;
  if constexpr (kTiled) {
    constexpr int kCols = kQuantThreads / 32;
    const int ktiles = (sl.groups_per_row + kCols - 1) / kCols;
    const int rt = (int)((unsigned)blockIdx.x / (unsigned)ktiles);
    col = ((int)blockIdx.x - rt * ktiles) * kCols + warp;
    row0 = (int64_t)rt * (U * kWarpGroups) + slot;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t row = row0 + u * kWarpGroups;
      ge[u] = row < tokens && col < sl.groups_per_row ? (row * sl.groups_per_row + col) * G : -1;
    }
  } else {
    const int64_t groups = tokens * sl.groups_per_row;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t g = ((int64_t)blockIdx.x * U + u) * (kUnitElems / G) + warp * kWarpGroups + slot;
      ge[u] = g < groups ? g * G : -1;
    }
  }
  uint4 raw[U][NCH];
#pragma unroll
  for (int u = 0; u < U; ++u) {
#pragma unroll
    for (int j = 0; j < NCH; ++j) raw[u][j] = make_uint4(0, 0, 0, 0);
    if (ge[u] >= 0) load_lane<NCH>(raw[u], x + ge[u] + l * kLaneElems, wide_in);
  }
  float my_scale = 0.f;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float v[kLaneElems];
#pragma unroll
    for (int j = 0; j < NCH; ++j) unpack_chunk<T>(raw[u][j], v + j * CE);
    uint32_t codes[NCH][CE / 4];
    const float scale = quant_group<T, LPG, kStdRange, NCH>(raw[u], v, eps, qmin, qmax, codes);
    if (l == u) my_scale = scale;
    if (ge[u] >= 0) store_lane(out_q + ge[u] + l * kLaneElems, &codes[0][0], wide_out);
  }
  if (l < U) {  // lane u of a group stores the scale of unit u
    int64_t e = ge[0];
#pragma unroll
    for (int u = 1; u < U; ++u)
      if (l == u) e = ge[u];
    if (e >= 0) {
      if constexpr (kTiled) {
        out_s[col * sl.stride_group + row0 + l * kWarpGroups] = my_scale;
      } else {
        const int64_t g = e / G;
        if (sl.contiguous) {
          out_s[g] = my_scale;
        } else {
          const int64_t t = div_groups(g, sl.groups_per_row);
          out_s[t * sl.stride_token + (g - t * sl.groups_per_row) * sl.stride_group] = my_scale;
        }
      }
    }
  }
}

// Fused silu_and_mul + quantizer.  x is [rows, 2d] (gate | up).  In the ring a tile is kTileElems consecutive OUTPUT
// elements of an expert's flat [rows, d] result, staged as one or more (gate, up) pairs of row
// segments.  h = T(T(silu(gate)) * up): silu in float32 rounded to T, then one packed multiply (the product of
// two 16-bit floats is exact in float32, so its single rounding equals rounding the float32 product), then
// the quantizer arithmetic on h in registers.
// Direct form: as the quantizer, 16 gate and 16 up values a thread and unit.
template <typename T, int LPG, int U>
__global__ void __launch_bounds__(kQuantThreads)
    silu_mul_quant_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q, float* __restrict__ out_s, int64_t rows,
                          int d, const int32_t* __restrict__ num_rows_dev, float eps, bool wide_in, bool wide_out,
                          bool trigger) {
  constexpr int CE = Chunk<T>::kElems, NCH = kLaneElems / CE, G = LPG * kLaneElems;
  if (trigger) ptx::launch_dependents();
  ptx::grid_dependency_wait();
  if (num_rows_dev != nullptr) {
    const int64_t lim = *num_rows_dev;
    rows = lim < rows ? lim : rows;
  }
  const int per_row = d / G, l = threadIdx.x % LPG;
  const int64_t groups = rows * per_row;
  const int64_t g0 = (int64_t)blockIdx.x * (U * (kUnitElems / G)) + threadIdx.x / LPG;
  if (g0 - threadIdx.x / LPG >= groups) return;  // the grid is sized from the host-side bound on rows
  uint4 graw[U][NCH], uraw[U][NCH];
#pragma unroll
  for (int u = 0; u < U; ++u) {
#pragma unroll
    for (int j = 0; j < NCH; ++j) graw[u][j] = uraw[u][j] = make_uint4(0, 0, 0, 0);
    const int64_t g = g0 + u * (kUnitElems / G);
    if (g < groups) {
      const T* gate = x + g * G + div_groups(g, per_row) * d + l * kLaneElems;
      load_lane<NCH>(graw[u], gate, wide_in);
      load_lane<NCH>(uraw[u], gate + d, wide_in);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    uint4 hraw[NCH];
    float v[kLaneElems];
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      float g[CE];
      unpack_chunk<T>(graw[u][j], g);
      const uint32_t up[4] = {uraw[u][j].x, uraw[u][j].y, uraw[u][j].z, uraw[u][j].w};
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = Packed2<T>::round_mul(silu_f32(g[2 * k]), silu_f32(g[2 * k + 1]), up[k]);
      hraw[j] = make_uint4(h[0], h[1], h[2], h[3]);
      unpack_chunk<T>(hraw[j], v + j * CE);
    }
    uint32_t codes[NCH][CE / 4];
    const float scale = quant_group<T, LPG, true, NCH>(hraw, v, eps, -448.0f, 448.0f, codes);
    const int64_t g = g0 + u * (kUnitElems / G);
    if (g < groups) {
      store_lane(out_q + g * G + l * kLaneElems, &codes[0][0], wide_out);
      if (l == 0) out_s[g] = scale;
    }
  }
}

// The quantizer of a MoE layer's activations, which go to expert-sorted rows: a warp quantises four groups of a token's row
// and writes their codes to every place the token has (512 bytes of each), so that no other launch copies rows.  The first
// `buckets` CTAs take a bucket of the sort each and zero its padding rows in the 32-row quadrant of its last block that also
// holds rows, the eight warps in turn.  (One warp a quadrant, of up to 31 rows, was as long as a small layer's whole launch:
// 2000 tokens of 1024 to two places 8.2 us of kernel, so 2.9; 1100 of 1152 8.1, so 3.1.)  Bound by HBM writes: 16384
// tokens of 2048 to eight places 58.6 us (5.7 TB/s), quantizer and gather 89.1; 4096 tokens of 7168 64.1 us, before 137.  With
// eight and sixteen groups a warp 58.6 and 60.9, 62.5 and 67.1.
template <typename T>
__global__ void __launch_bounds__(kQuantThreads)
    quant_sorted_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q, float* __restrict__ out_s,
                        const int32_t* __restrict__ inverse, const int32_t* __restrict__ sorted_ids,
                        const int32_t* __restrict__ starts, int64_t items, int buckets, int pieces, int groups, int topk,
                        int64_t numel, float eps, bool wide_in) {
  constexpr int LPG = 8, CE = 8, NCH = 2, G = 128, kBlock = 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ptx::grid_dependency_wait();
  ptx::launch_dependents();
  const int64_t hidden = (int64_t)groups * G;
  if ((int)blockIdx.x < buckets) {
    const int stop = starts[blockIdx.x + 1];
    if (starts[blockIdx.x] == stop) return;
    // (a bucket's rows come first, and only its last block has padding)
    const int held = __syncthreads_count(threadIdx.x < kBlock && sorted_ids[stop - kBlock + (int)threadIdx.x] < numel);
    for (int r = stop - kBlock + held + warp; r < stop - kBlock + (held + 31) / 32 * 32; r += kQuantThreads / 32) {
      uint8_t* q = out_q + r * hidden;
      for (int c = lane * 16; c < (int)hidden; c += 512) *reinterpret_cast<uint4*>(q + c) = make_uint4(0, 0, 0, 0);
      for (int g = lane; g < groups; g += 32) out_s[(int64_t)r * groups + g] = 0.f;
    }
    return;
  }
  const int64_t it = (int64_t)(blockIdx.x - buckets) * (kQuantThreads / 32) + warp;
  if (it >= items) return;
  const int64_t t = it / pieces;
  const int g = (int)(it - t * pieces) * (32 / LPG) + lane / LPG, l = lane % LPG;
  const bool on = g < groups;
  uint4 raw[NCH] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  if (on) load_lane<NCH>(raw, x + t * hidden + g * G + l * kLaneElems, wide_in);
  int place = lane < topk ? inverse[t * topk + lane] : -1;
  float v[kLaneElems];
#pragma unroll
  for (int j = 0; j < NCH; ++j) unpack_chunk<T>(raw[j], v + j * CE);
  uint32_t codes[NCH][CE / 4];
  const float scale = quant_group<T, LPG, true, NCH>(raw, v, eps, -448.0f, 448.0f, codes);
  const uint4 out = make_uint4(codes[0][0], codes[0][1], codes[1][0], codes[1][1]);
  for (int k = 0; k < topk; ++k) {
    if ((k & 31) == 0 && k > 0) place = k + lane < topk ? inverse[t * topk + k + lane] : -1;
    const int64_t r = __shfl_sync(0xffffffffu, place, k & 31);
    if (r < 0 || !on) continue;
    *reinterpret_cast<uint4*>(out_q + r * hidden + g * G + l * kLaneElems) = out;
    if (l == 0) out_s[r * groups + g] = scale;
  }
}

constexpr int kSiluStages = 2;  // 2 x (16 KB gate + 16 KB up) per CTA, three CTAs per SM (80 registers)

constexpr int kMaskedMaxExperts = 1024;  // experts of one masked call (four per thread in the tile count scan)

// Masked form: the input is [experts, rows_per_expert, 2d] and only the first masked_m[e] rows of expert e are valid
// (the layout of python/sglang/srt/layers/moe/ep_moe/kernels.py:287-361).  The valid rows of every expert are cut
// into tiles of their own, numbered one expert after the other; rows beyond masked_m[e] are neither read nor written.
template <typename T, int LPG>
__global__ void __launch_bounds__(kStreamThreads, 3)
    silu_mul_quant_masked_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q, float* __restrict__ out_s,
                                 int d, float eps, float qmin, float qmax, uint32_t probes,
                                 const int32_t* __restrict__ masked_m, int num_experts, int64_t rows_per_expert) {
  static_assert(sizeof(T) == 2, "16-bit inputs only");
  constexpr int CE = 8, NCH = 4, GC = LPG * NCH, G = LPG * kThreadElems;
  constexpr uint32_t kHalfBytes = kTileElems * 2;  // gate part of a stage; the up part follows it
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kSiluStages];
  __shared__ int s_abort;
  __shared__ int s_tiles_before[kMaskedMaxExperts + 1];  // tiles of the experts before e
  __shared__ int s_warp_sum[kStreamThreads / 32];
  ptx::grid_dependency_wait();
  const uint32_t smem_base = ptx::smem_u32(smem_raw);
  const int tid = threadIdx.x;
  auto valid_rows = [&](int e) -> int64_t {
    const int64_t m = masked_m[e];
    return m < 0 ? 0 : (m > rows_per_expert ? rows_per_expert : m);
  };
  // exclusive scan of the experts' tile counts: four experts per thread, then the warps' sums
  int cnt[4], mine = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = tid * 4 + k;
    cnt[k] = e < num_experts ? (int)((valid_rows(e) * d + kTileElems - 1) / kTileElems) : 0;
    mine += cnt[k];
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if ((tid & 31) >= o) incl += up;
  }
  if ((tid & 31) == 31) s_warp_sum[tid >> 5] = incl;
  __syncthreads();
  int before = incl - mine;
  for (int w = 0; w < (tid >> 5); ++w) before += s_warp_sum[w];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = tid * 4 + k;
    if (e < num_experts) s_tiles_before[e] = before;
    before += cnt[k];
  }
  if (tid == kStreamThreads - 1) s_tiles_before[num_experts] = before;  // (experts beyond num_experts count 0)
  __syncthreads();
  const int64_t tiles = s_tiles_before[num_experts];
  if ((int64_t)blockIdx.x >= tiles) return;  // the grid is sized from the host-side bound on rows
  const int64_t my_tiles = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;

  // tile i of this CTA: first element within its expert, that range's element count, and
  // the range's first row
  auto locate = [&](int64_t i, int64_t& e0, int64_t& lim, int64_t& row_base) {
    const int64_t gt = blockIdx.x + i * gridDim.x;
    int lo = 0, hi = num_experts;  // the expert with s_tiles_before[e] <= gt < s_tiles_before[e + 1]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((int64_t)s_tiles_before[mid] <= gt) lo = mid; else hi = mid;
    }
    e0 = (gt - s_tiles_before[lo]) * (int64_t)kTileElems;
    lim = valid_rows(lo) * d;
    row_base = (int64_t)lo * rows_per_expert;
  };

  auto issue = [&](int64_t i) {  // thread 0 only
    const int slot = (int)(i % kSiluStages);
    int64_t e0, lim, row_base;
    locate(i, e0, lim, row_base);
    const int64_t left = lim - e0;
    const int n = left >= kTileElems ? kTileElems : (int)left;
    const uint32_t bar = ptx::smem_u32(&bars[slot]);
    const uint32_t dst = smem_base + slot * (2 * kHalfBytes);
    ptx::mbar_arrive_expect_tx(bar, (uint32_t)n * 4u);
    int64_t r = e0 / d;
    int c = (int)(e0 - r * d);
    r += row_base;
    for (int off = 0; off < n;) {
      const int seg = (d - c) < (n - off) ? (d - c) : (n - off);
      const T* row = x + r * 2 * (int64_t)d + c;
      bulk_load_1d(dst + off * 2, row, (uint32_t)seg * 2u, bar);
      bulk_load_1d(dst + kHalfBytes + off * 2, row + d, (uint32_t)seg * 2u, bar);
      off += seg;
      c = 0;
      ++r;
    }
  };

  if (tid == 0) {
    s_abort = 0;
#pragma unroll
    for (int s = 0; s < kSiluStages; ++s) ptx::mbar_init(ptx::smem_u32(&bars[s]), 1);
    ptx::mbar_fence_init();
    for (int64_t i = 0; i < kSiluStages && i < my_tiles; ++i) issue(i);
  }
  __syncthreads();

  const int g_local = tid / LPG, l = tid % LPG;
  const int rot = chunk_rotation<T, LPG>(g_local);
  int cj[NCH];
#pragma unroll
  for (int j = 0; j < NCH; ++j) cj[j] = (LPG * j + l + rot) % GC;

  for (int64_t i = 0; i < my_tiles; ++i) {
    const int slot = (int)(i % kSiluStages);
    const uint32_t parity = (uint32_t)((i / kSiluStages) & 1);
    if (!ptx::mbar_probe(ptx::smem_u32(&bars[slot]), parity, probes)) s_abort = 1;
    uint4 graw[NCH], uraw[NCH];
    const uint32_t src = smem_base + slot * (2 * kHalfBytes) + (uint32_t)(g_local * GC) * 16u;
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      graw[j] = ptx::lds_128(src + (uint32_t)cj[j] * 16u);
      uraw[j] = ptx::lds_128(src + kHalfBytes + (uint32_t)cj[j] * 16u);
    }
    __syncthreads();  // the slot is in registers and can be refilled
    if (s_abort) {  // (uniform: read after the barrier)
      stream_give_up(tid);
      return;
    }
    if (tid == 0 && i + kSiluStages < my_tiles) issue(i + kSiluStages);

    uint4 hraw[NCH];
    float v[NCH * CE];
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      float g[CE];
      unpack_chunk<T>(graw[j], g);
      const uint32_t up[4] = {uraw[j].x, uraw[j].y, uraw[j].z, uraw[j].w};
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = Packed2<T>::round_mul(silu_f32(g[2 * k]), silu_f32(g[2 * k + 1]), up[k]);
      hraw[j] = make_uint4(h[0], h[1], h[2], h[3]);
      unpack_chunk<T>(hraw[j], v + j * CE);
    }
    uint32_t codes[NCH][CE / 4];
    const float scale = quant_group<T, LPG, true>(hraw, v, eps, qmin, qmax, codes);

    int64_t e0, lim, row_base;
    locate(i, e0, lim, row_base);
    const int64_t ge_in = e0 + (int64_t)g_local * G;
    if (ge_in < lim) {
      const int64_t ge = row_base * d + ge_in;
#pragma unroll
      for (int j = 0; j < NCH; ++j)
        *reinterpret_cast<uint2*>(out_q + ge + cj[j] * CE) = make_uint2(codes[j][0], codes[j][1]);
      if (l == 0) out_s[ge / G] = scale;
    }
  }
}

inline bool aligned_to(const void* p, uintptr_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

template <typename T, int LPG, bool kStd>
static int launch_quant_ring(const void* input, void* output_q, float* output_s, int64_t total_elems,
                             const ScaleLayout& sl, float eps, float qmin, float qmax, bool trigger,
                             cudaStream_t stream) {
  constexpr size_t smem = (size_t)kStagesOf<T> * kTileElems * sizeof(T);
  auto kern = quant_stream_kernel<T, LPG, kStd>;
  // opt in to the ring's dynamic shared memory (a per-function, per-device attribute; cheap to repeat)
  SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t tiles = (total_elems + kTileElems - 1) / kTileElems;
  const int64_t resident = (int64_t)sm_count() * (sizeof(T) == 4 ? 2 : 3);
  const unsigned grid = (unsigned)(tiles < resident ? tiles : resident);
  SGLB_CUDA(launch_pdl(kern, grid, kStreamThreads, smem, stream, static_cast<const T*>(input), static_cast<uint8_t*>(output_q), output_s,
                                               total_elems, sl.groups_per_row, sl.stride_token, sl.stride_group,
                                               sl.contiguous, eps, qmin, qmax, g_stream_wait_probes, trigger));
  return SGLB200_OK;
}

template <typename T, int LPG, bool kStd>
static int launch_quant_inst(const void* input, void* output_q, float* output_s, int64_t tokens, const ScaleLayout& sl,
                             float eps, float qmin, float qmax, bool trigger, cudaStream_t stream) {
  constexpr int G = LPG * kLaneElems;
  const int64_t groups = tokens * sl.groups_per_row;
  const bool wide_in = aligned_to(input, 32), wide_out = aligned_to(output_q, 16);
  auto go = [&](auto kern, int64_t blocks) -> int {
    SGLB_REQUIRE(blocks < (1ll << 31), "quantizer: input too large");
    SGLB_CUDA(launch_pdl(kern, (unsigned)blocks, kQuantThreads, 0, stream, static_cast<const T*>(input),
                         static_cast<uint8_t*>(output_q), output_s, tokens, sl, eps, qmin, qmax, wide_in, wide_out, trigger));
    return SGLB200_OK;
  };
  const int64_t elems = groups * G, sms = sm_count();
  // The flat direct form requests a CTA's whole input at once and sets nothing up for it; the ring's deeper staging wins
  // where 16-bit inputs are many times what the SMs hold.  With dense row-major scales: 64 x 7168 bf16 1.8 us, ring 2.4;
  // 781 x 4096 2.6 and 3.4; 2441 x 4096 5.6 and 5.9; 4882 x 4096 (33 CTAs an SM) 9.8 and 9.8; 7080 x 4096 14.9 and 13.8;
  // 8192 x 18432 84.4 and 73.9; groups of 32 to 256 and fp16 cross between 30 and 65 CTAs an SM.  float32, whose ring has
  // two CTAs an SM, never crosses: 585 x 4096 2.4 and 2.8, 8192 x 18432 106.4 and 129.7.  Other layouts leave the flat
  // form earlier: its scales then go out one word per sector.  A limit on the ring's waits (the tests of its give-up)
  // selects the ring at any size.
  const bool ring = g_stream_wait_probes != ptx::kProbeLimit;
  const bool flat = elems <= sms * (sl.contiguous ? 32 : 4) * kUnitElems || (sl.contiguous && sizeof(T) == 4);
  if (!ring && flat)
    return go(quant_kernel<T, LPG, kStd, 1, false>, (elems + kUnitElems - 1) / kUnitElems);
  // M-major scales, up to 32 CTA-units an SM: the tiled direct form (1024 x 4096: 3.5 us, ring 4.0; 2048 x 4096: 5.2 and
  // 6.0; 4096 x 4096: 9.0 and 10.1).  Its warps idle in the last tile of a row: not where that is more than a quarter.
  const int64_t ktiles = (sl.groups_per_row + 7) / 8, tile_rows = 2 * (32 / LPG);
  if (!ring && !sl.contiguous && sl.stride_token == 1 && sl.groups_per_row >= ktiles * 6 && elems <= sms * 32 * kUnitElems)
    return go(quant_kernel<T, LPG, kStd, 2, true>, ktiles * ((tokens + tile_rows - 1) / tile_rows));
  return launch_quant_ring<T, LPG / 2, kStd>(input, output_q, output_s, elems, sl, eps, qmin, qmax, trigger, stream);
}

template <typename T>
static int launch_quant_sorted(const void* x, void* out_q, float* out_s, const int32_t* inverse, const int32_t* sorted_ids,
                               const int32_t* starts, int buckets, int64_t tokens, int topk, int64_t hidden, float eps,
                               cudaStream_t st) {
  constexpr int kWarps = kQuantThreads / 32;
  const int groups = (int)(hidden / 128), pieces = (groups + 3) / 4;
  const int64_t items = tokens * pieces, row_ctas = (items + kWarps - 1) / kWarps;
  SGLB_REQUIRE(row_ctas + buckets < (1ll << 31), "quantizer: input too large");
  SGLB_CUDA(launch_pdl(quant_sorted_kernel<T>, (unsigned)(row_ctas + buckets), kQuantThreads, 0, st, static_cast<const T*>(x),
                       static_cast<uint8_t*>(out_q), out_s, inverse, sorted_ids, starts, items, buckets, pieces,
                       groups, topk, tokens * topk, eps, aligned_to(x, 32)));
  return SGLB200_OK;
}

template <typename T>
static int launch_quant(const void* input, void* output_q, float* output_s, int64_t num_tokens, int64_t hidden,
                        int group_size, float eps, float qmin, float qmax, int64_t s_stride_token,
                        int64_t s_stride_group, bool trigger, cudaStream_t stream) {
  const int groups_per_row = (int)(hidden / group_size);
  const ScaleLayout sl{groups_per_row, s_stride_token, s_stride_group,
                       s_stride_group == 1 && s_stride_token == groups_per_row};
  const bool std_range = (qmin == -448.0f && qmax == 448.0f);
#define SGLB_LAUNCH_Q(LPG)                                                                                        \
  return std_range ? launch_quant_inst<T, LPG, true>(input, output_q, output_s, num_tokens, sl, eps, qmin, qmax,  \
                                                     trigger, stream)                                             \
                   : launch_quant_inst<T, LPG, false>(input, output_q, output_s, num_tokens, sl, eps, qmin, qmax, \
                                                      trigger, stream)
  switch (group_size) {
    case 32: SGLB_LAUNCH_Q(2);
    case 64: SGLB_LAUNCH_Q(4);
    case 128: SGLB_LAUNCH_Q(8);
    case 256: SGLB_LAUNCH_Q(16);
    default: return fail(SGLB200_E_INVALID, "quantizer: group_size %d not in {32,64,128,256}", group_size);
  }
#undef SGLB_LAUNCH_Q
}

template <typename T, int LPG>
static int launch_silu_mul_quant_inst(const void* input, void* output_q, float* output_s, int64_t rows, int64_t d,
                                      float eps, const int32_t* num_rows_dev, bool trigger, cudaStream_t stream) {
  // Two units a thread from 32 CTA-units an SM on: more loads in flight where occupancy no longer grows (131072 x 768
  // bf16: 89 us, one unit 95, staged by bulk copies 104; 8192 x 3584: 29.0, 29.9 and 29.4), one below (256 x 768: 2.0, 2.9
  // and 4.1; 16384 x 768: 12.2, 12.7 and 15.6; 1999 x 3584: 7.6, 7.8 and 8.5).
  const int units = rows * d > (int64_t)sm_count() * 32 * kUnitElems ? 2 : 1;
  const int64_t per = (int64_t)units * kUnitElems, blocks = (rows * d + per - 1) / per;
  SGLB_REQUIRE(blocks < (1ll << 31), "silu_mul_quant: input too large");
  SGLB_CUDA(launch_pdl(units == 2 ? silu_mul_quant_kernel<T, LPG, 2> : silu_mul_quant_kernel<T, LPG, 1>, (unsigned)blocks,
                       kQuantThreads, 0, stream, static_cast<const T*>(input), static_cast<uint8_t*>(output_q), output_s,
                       rows, (int)d, num_rows_dev, eps, aligned_to(input, 32), aligned_to(output_q, 16), trigger));
  return SGLB200_OK;
}

template <typename T, int LPG>
static int launch_silu_mul_quant_masked_inst(const void* input, void* output_q, float* output_s, int num_experts,
                                             int64_t rows_per_expert, int64_t d, float eps, const int32_t* masked_m,
                                             cudaStream_t stream) {
  constexpr size_t smem = (size_t)kSiluStages * 2 * kTileElems * sizeof(T);
  auto kern = silu_mul_quant_masked_kernel<T, LPG>;
  SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // (every expert's last tile may be partial, so the bound counts the experts' tiles one by one)
  const int64_t tiles = (int64_t)num_experts * ((rows_per_expert * d + kTileElems - 1) / kTileElems);
  const int64_t resident = (int64_t)sm_count() * 3;
  SGLB_CUDA(launch_pdl(kern, (unsigned)(tiles < resident ? tiles : resident), kStreamThreads, smem, stream,
                       static_cast<const T*>(input), static_cast<uint8_t*>(output_q), output_s, (int)d, eps, -448.0f, 448.0f,
                       g_stream_wait_probes, masked_m, num_experts, rows_per_expert));
  return SGLB200_OK;
}

template <typename T>
static int launch_silu_mul_quant(const void* input, void* output_q, float* output_s, int64_t rows, int64_t d,
                                 int group_size, float eps, const int32_t* num_rows_dev, bool trigger, cudaStream_t stream) {
  if (rows * d == 0) return SGLB200_OK;
  SGLB_REQUIRE(d < (1ll << 30), "silu_mul_quant: d %lld too large", (long long)d);
  switch (group_size) {
    case 32: return launch_silu_mul_quant_inst<T, 2>(input, output_q, output_s, rows, d, eps, num_rows_dev, trigger, stream);
    case 64: return launch_silu_mul_quant_inst<T, 4>(input, output_q, output_s, rows, d, eps, num_rows_dev, trigger, stream);
    case 128: return launch_silu_mul_quant_inst<T, 8>(input, output_q, output_s, rows, d, eps, num_rows_dev, trigger, stream);
    case 256: return launch_silu_mul_quant_inst<T, 16>(input, output_q, output_s, rows, d, eps, num_rows_dev, trigger, stream);
    default: return fail(SGLB200_E_INVALID, "silu_mul_quant: group_size %d not in {32,64,128,256}", group_size);
  }
}

template <typename T>
static int launch_silu_mul_quant_masked(const void* input, void* output_q, float* output_s, int num_experts,
                                        int64_t rows_per_expert, int64_t d, int group_size, float eps,
                                        const int32_t* masked_m, cudaStream_t stream) {
#define SGLB_MASKED(LPG)                                                                                         \
  return launch_silu_mul_quant_masked_inst<T, LPG>(input, output_q, output_s, num_experts, rows_per_expert, d, eps, \
                                                   masked_m, stream)
  switch (group_size) {
    case 32: SGLB_MASKED(1);
    case 64: SGLB_MASKED(2);
    case 128: SGLB_MASKED(4);
    case 256: SGLB_MASKED(8);
    default: return fail(SGLB200_E_INVALID, "silu_mul_quant: group_size %d not in {32,64,128,256}", group_size);
  }
#undef SGLB_MASKED
}

}  // namespace sglb200

using namespace sglb200;

extern "C" int sglb200_silu_and_mul_masked_quant_fp8(const void* input, int dtype, void* output_q, float* output_s,
                                                     int num_experts, int64_t rows_per_expert, int64_t d,
                                                     int group_size, float eps, const int32_t* masked_m,
                                                     void* stream) {
  SGLB_REQUIRE(num_experts >= 0 && num_experts <= kMaskedMaxExperts && rows_per_expert >= 0 && d > 0 &&
                   group_size > 0 && d % group_size == 0 && d < (1ll << 30),
               "silu_mul_masked_quant: bad shape experts=%d (at most %d) rows_per_expert=%lld d=%lld group=%d",
               num_experts, kMaskedMaxExperts, (long long)rows_per_expert, (long long)d, group_size);
  if (num_experts == 0 || rows_per_expert == 0) return SGLB200_OK;
  SGLB_REQUIRE(rows_per_expert * d < (1ll << 40), "silu_mul_masked_quant: expert of %lld x %lld elements too large",
               (long long)rows_per_expert, (long long)d);
  SGLB_REQUIRE(input && output_q && output_s && masked_m, "silu_mul_masked_quant: null pointer");
  SGLB_REQUIRE(aligned16(input) && (reinterpret_cast<uintptr_t>(output_q) & 7u) == 0,
               "silu_mul_masked_quant: input must be 16-byte and output_q 8-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case 0:
      return launch_silu_mul_quant_masked<__nv_bfloat16>(input, output_q, output_s, num_experts, rows_per_expert, d,
                                                         group_size, eps, masked_m, st);
    case 1:
      return launch_silu_mul_quant_masked<__half>(input, output_q, output_s, num_experts, rows_per_expert, d,
                                                  group_size, eps, masked_m, st);
    default:
      return fail(SGLB200_E_UNSUPPORTED, "silu_mul_masked_quant: dtype code %d (0 bf16, 1 fp16)", dtype);
  }
}

int sglb200::quant_fp8(const void* input, int in_dtype, void* output_q, float* output_s,
                                                 int64_t num_tokens, int64_t hidden, int group_size, float eps,
                                                 float fp8_min, float fp8_max, int64_t s_stride_token,
                                                 int64_t s_stride_group, bool trigger, cudaStream_t st) {
  SGLB_REQUIRE(num_tokens >= 0 && hidden > 0, "quantizer: bad shape [%lld, %lld]", (long long)num_tokens,
               (long long)hidden);
  SGLB_REQUIRE(group_size > 0 && hidden % group_size == 0, "quantizer: hidden %lld not divisible by group_size %d",
               (long long)hidden, group_size);
  if (num_tokens == 0) return SGLB200_OK;
  SGLB_REQUIRE(input && output_q && output_s, "quantizer: null pointer");
  SGLB_REQUIRE(aligned16(input) && (reinterpret_cast<uintptr_t>(output_q) & 7u) == 0,
               "quantizer: input must be 16-byte and output_q 8-byte aligned");
  switch (in_dtype) {
    case 0:
      return launch_quant<__nv_bfloat16>(input, output_q, output_s, num_tokens, hidden, group_size, eps, fp8_min,
                                         fp8_max, s_stride_token, s_stride_group, trigger, st);
    case 1:
      return launch_quant<__half>(input, output_q, output_s, num_tokens, hidden, group_size, eps, fp8_min, fp8_max,
                                  s_stride_token, s_stride_group, trigger, st);
    case 2:
      return launch_quant<float>(input, output_q, output_s, num_tokens, hidden, group_size, eps, fp8_min, fp8_max,
                                 s_stride_token, s_stride_group, trigger, st);
    default:
      return fail(SGLB200_E_UNSUPPORTED, "quantizer: dtype code %d (0 bf16, 1 fp16, 2 fp32)", in_dtype);
  }
}

int sglb200::quant_sorted(const void* x, int dtype, void* out_q, float* out_s, const int32_t* inverse, const int32_t* sorted_ids,
                          const int32_t* starts, int buckets, int64_t tokens, int topk, int64_t hidden, float eps,
                          cudaStream_t st) {
  SGLB_REQUIRE(aligned16(x), "quantizer: input must be 16-byte aligned");
  return dtype == 0 ? launch_quant_sorted<__nv_bfloat16>(x, out_q, out_s, inverse, sorted_ids, starts, buckets, tokens, topk,
                                                         hidden, eps, st)
                    : launch_quant_sorted<__half>(x, out_q, out_s, inverse, sorted_ids, starts, buckets, tokens, topk, hidden,
                                                  eps, st);
}

extern "C" int sglb200_per_token_group_quant_fp8(const void* input, int in_dtype, void* output_q, float* output_s,
                                                 int64_t num_tokens, int64_t hidden, int group_size, float eps,
                                                 float fp8_min, float fp8_max, int64_t s_stride_token,
                                                 int64_t s_stride_group, void* stream) {
  return quant_fp8(input, in_dtype, output_q, output_s, num_tokens, hidden, group_size, eps, fp8_min, fp8_max, s_stride_token,
                   s_stride_group, false, static_cast<cudaStream_t>(stream));
}

int sglb200::silu_mul_quant_fp8(const void* input, int dtype, void* output_q, float* output_s,
                                              int64_t rows, int64_t d, int group_size, float eps,
                                              const int32_t* num_rows_dev, bool trigger, cudaStream_t st) {
  SGLB_REQUIRE(rows >= 0 && d > 0 && group_size > 0 && d % group_size == 0,
               "silu_mul_quant: bad shape rows=%lld d=%lld group=%d", (long long)rows, (long long)d, group_size);
  if (rows == 0) return SGLB200_OK;
  SGLB_REQUIRE(input && output_q && output_s, "silu_mul_quant: null pointer");
  SGLB_REQUIRE(aligned16(input) && (reinterpret_cast<uintptr_t>(output_q) & 7u) == 0,
               "silu_mul_quant: input must be 16-byte and output_q 8-byte aligned");
  switch (dtype) {
    case 0:
      return launch_silu_mul_quant<__nv_bfloat16>(input, output_q, output_s, rows, d, group_size, eps, num_rows_dev,
                                                  trigger, st);
    case 1:
      return launch_silu_mul_quant<__half>(input, output_q, output_s, rows, d, group_size, eps, num_rows_dev, trigger, st);
    default:
      return fail(SGLB200_E_UNSUPPORTED, "silu_mul_quant: dtype code %d (0 bf16, 1 fp16)", dtype);
  }
}

extern "C" int sglb200_silu_and_mul_quant_fp8(const void* input, int dtype, void* output_q, float* output_s,
                                              int64_t rows, int64_t d, int group_size, float eps,
                                              const int32_t* num_rows_dev, void* stream) {
  return silu_mul_quant_fp8(input, dtype, output_q, output_s, rows, d, group_size, eps, num_rows_dev, false,
                            static_cast<cudaStream_t>(stream));
}

extern "C" void sglb200_stream_set_wait_probes(uint32_t probes) {
  g_stream_wait_probes = probes == 0 ? ptx::kProbeLimit : probes;
}

extern "C" int sglb200_stream_status_clear(void) {
  const int zero = 0;
  SGLB_CUDA(cudaMemcpyToSymbol(g_stream_status, &zero, sizeof(int)));
  return SGLB200_OK;
}

extern "C" int sglb200_stream_status(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_stream_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
