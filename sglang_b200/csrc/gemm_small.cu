// Quantise + multiply in one launch, for linear layers on at most 16 activation rows whose weights are so small that
// latency is all there is:
//
//   C[m,n] = out_t( sum_kb a_s[m,kb] * b_s[n/128,kb] * sum_{k in kb} q(x)[m,k] * B[n,k] ) (+ bias)
//
// A decoded token through a 2112 x 7168 layer is 2.3 us of HBM time.  As quantizer + GEMM it took 8.5 us: two launches, a
// round trip of the codes through L2, a ring with per-slab hand-offs; in one launch 5.7 us.  The CTAs of a
// cluster share K and each holds its few slabs whole: one thread requests all of its weight tiles as soon as the kernel
// before is complete (0.1 to 0.5 us later than at the start of the launch, which is not safe: that kernel may have
// written them; asking for them towards L2 at the start gained nothing), meanwhile the other warps quantise the CTA's part
// of the activations straight into the swizzled MMA operand (every CTA of the same K range repeats that for itself: a few
// kilobytes; with 64 rows it cost more than the launch it saves, 14.1 against 12.3 us), every slab has an accumulator of
// its own, and there is one barrier between each two steps.  The cluster adds its partial sums through distributed
// shared memory.  Operands as in gemm_rows.cu: weights on the M side, activation rows on the N side.
#include <cuda.h>

#include "common.cuh"
#include "gemm_rows.cuh"
#include "quant_math.cuh"

namespace sglb200 {

constexpr int kSmallRows = 16;
constexpr int kSmallWarps = 8;                            // quantise (the first four then promote); one more loads and multiplies
constexpr int kSmallThreads = (kSmallWarps + 1) * 32;
constexpr int kSmallMaxSlabs = 8;
constexpr int kSmallTmem = kSmallMaxSlabs * kSmallRows;
constexpr uint32_t kSmallTokBytes = kSmallRows * kRowsBK;
constexpr int64_t kSmallSmem = 111 * 1024;                // two CTAs per SM
constexpr float kSmallEps = 1e-10f;                       // as the quantizer of a linear layer

struct SmallCtl {
  uint64_t w_full[kSmallMaxSlabs];
  uint64_t tok_full, acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ int g_small_status = 0;  // 0 ok, 1 = a pipeline wait expired

template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 2)
    fp8_small_linear_kernel(const __grid_constant__ CUtensorMap map_w, const T* __restrict__ x, int64_t K, int max_slabs,
                            const RowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* weights = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tokens = weights + max_slabs * kWBytes;
  float* sc = reinterpret_cast<float*>(tokens + max_slabs * kSmallTokBytes);  // [slab][row]: a_s * b_s
  SmallCtl* ctl = reinterpret_cast<SmallCtl*>(sc + max_slabs * kSmallRows);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &ctl->abort_flag;
  const int splits = p.splits, rank = (int)(blockIdx.x % splits), n_tile = (int)(blockIdx.x / splits);
  const int kb_begin = rank * p.kb_total / splits, slabs = (rank + 1) * p.kb_total / splits - kb_begin;

  ptx::launch_dependents();
  if (warp == kSmallWarps) {
    if (lane == 0) {
      for (int s = 0; s < slabs; ++s) ptx::mbar_init(ptx::smem_u32(&ctl->w_full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&ctl->tok_full), kSmallWarps * 32);
      ptx::mbar_init(ptx::smem_u32(&ctl->acc_full), 1);
      ctl->abort_flag = 0;
      ptx::mbar_fence_init();
    }
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), kSmallTmem);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base, bar_tok = ptx::smem_u32(&ctl->tok_full), bar_acc = ptx::smem_u32(&ctl->acc_full);

  if (warp == kSmallWarps) {
    // ------------------------------ MMA issuer ------------------------------
    if (ptx::elect_one()) {
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // see gemm.cu
      constexpr uint32_t idesc = ptx::make_idesc_e4m3_f32(kRowsBM, kSmallRows);
      const uint32_t w_lo = ((ptx::smem_u32(weights) & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t t_lo = ((ptx::smem_u32(tokens) & 0x3ffffu) >> 4) | (1u << 16);
      // The weights too are read only after the wait: the kernel before this one may have written them, and a launch that
      // may start early can start before such writes are visible even where that kernel triggers nothing.
      ptx::grid_dependency_wait();
      for (int s = 0; s < slabs; ++s) {
        const uint32_t bar = ptx::smem_u32(&ctl->w_full[s]);
        ptx::mbar_arrive_expect_tx(bar, kWBytes);
        ptx::tma_load_3d(ptx::smem_u32(weights) + s * kWBytes, &map_w, bar, (kb_begin + s) * kRowsBK, n_tile * kRowsBM, 0);
      }
      bool ok = ROWS_WAIT(bar_tok, 0);
      for (int s = 0; s < slabs && ok; ++s) {
        ok = ROWS_WAIT(ptx::smem_u32(&ctl->w_full[s]), 0);
        if (!ok) break;
        ptx::tc_fence_after();
        const uint32_t a_lo = w_lo + s * (kWBytes >> 4), b_lo = t_lo + s * (kSmallTokBytes >> 4);
#pragma unroll
        for (int k = 0; k < kRowsBK / 32; ++k)
          ptx::mma_f8f6f4(tmem_base + s * kSmallRows, ptx::pack_f32x2(a_lo + 2 * k, kDescHi), ptx::pack_f32x2(b_lo + 2 * k, kDescHi),
                          idesc, k > 0 ? 1u : 0u);
      }
      if (ok) ptx::mma_commit(bar_acc);
      else *abort_flag = 1;
    }
    __syncwarp();
  } else {
    // ------------------------------ quantise this CTA's activations ------------------------------
    // Four lanes per (row, slab) group, eight groups per warp and step, rows fastest (their swizzled places differ in
    // banks).  Rows past M are neither read nor written: what lies there is multiplied into columns that nobody reads.  With all
    // sixteen quantised, one row and more than four slabs took two steps, one round trip to memory after the other: 1 x 2112 x
    // 7168 6.70 us, so 5.66; 8 x 2112 x 7168 7.27 -> 6.48; up to four slabs and sixteen rows alike.  (Asking for the second step's
    // activations before the first is quantised: 16 x 2112 x 7168 7.8 -> 8.2.)
    const int l = lane & 3, total = (int)p.M * slabs;
    const float* b_row = p.b_s + (int64_t)n_tile * p.kb_total + kb_begin;
    ptx::grid_dependency_wait();
    for (int g0 = warp * 8; g0 < total; g0 += kSmallWarps * 8) {  // (uniform over the warp)
      const int g = min(g0 + (lane >> 2), total - 1);  // (lanes past the last group do as the last)
      const int slab = (int)((uint32_t)g * p.per_row >> 16), row = g - slab * (int)p.M;
      const T* src = x + (int64_t)row * K + (kb_begin + slab) * kRowsBK + l * 8;
      uint4 raw[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) raw[j] = ld_nc_16(src + j * 32);
      const float bs = __ldg(b_row + slab);
      float v[32];
#pragma unroll
      for (int j = 0; j < 4; ++j) unpack_chunk<T>(raw[j], v + j * 8);
      uint32_t codes[4][2];
      const float scale = quant_group<T, 4, true>(raw, v, kSmallEps, -448.0f, 448.0f, codes);
      const uint32_t dst = ptx::smem_u32(tokens) + slab * kSmallTokBytes + row * kRowsBK;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = 4 * j + l;  // 8-byte piece of the row
        ptx::sts_64(dst + ((((uint32_t)c >> 1) ^ (row & 7)) << 4) + (c & 1) * 8, codes[j][0], codes[j][1]);
      }
      if (l == 0) sc[slab * kSmallRows + row] = scale * bs;
    }
    ptx::fence_async_smem();
    ptx::mbar_arrive(bar_tok);
    // ------------------------------ promotion ------------------------------
    if (warp < 4) {
      if (!ROWS_WAIT(bar_tok, 0) || !ROWS_WAIT(bar_acc, 0)) {
        *abort_flag = 1;
      } else {
        ptx::tc_fence_after();
        float acc[kSmallRows];
#pragma unroll
        for (int j = 0; j < kSmallRows; ++j) acc[j] = 0.f;
        for (int s = 0; s < slabs; ++s) {
          uint32_t r[kSmallRows];
          ptx::tmem_ld_32x16(tmem_base + ((uint32_t)(warp * 32) << 16) + s * kSmallRows, r);
          ptx::tmem_ld_wait();
          const float4* s4 = reinterpret_cast<const float4*>(sc + s * kSmallRows);
#pragma unroll
          for (int j = 0; j < kSmallRows; j += 4) {
            const float4 f = s4[j / 4];
            ptx::fma2(acc[j], acc[j + 1], r[j], r[j + 1], f.x, f.y);
            ptx::fma2(acc[j + 2], acc[j + 3], r[j + 2], r[j + 3], f.z, f.w);
          }
        }
        // partial sums [column][weight row] over the weights, which have been consumed
        float* part = reinterpret_cast<float*>(weights) + warp * 32 + lane;
#pragma unroll
        for (int j = 0; j < kSmallRows; ++j) part[j * kPartPitch] = acc[j];
      }
    }
  }

  // ------------------------------ sum over the CTAs of the cluster ------------------------------
  __syncwarp();
  ptx::cluster_sync();
  const RowsTile t{n_tile, 0, kSmallRows, 0};
  if (ctl->abort_flag == 0) rows_cluster_sum<kMostClusterCtas>(p, t, rank, ptx::smem_u32(weights), tid, kSmallThreads);
  ptx::cluster_sync();  // no CTA leaves while another reads its shared memory

  // ------------------------------ teardown ------------------------------
  ptx::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag != 0 && tid == 0) {
    atomicExch(&g_small_status, 1);
    // give TMA copies that may still be in flight time to land before the CTA's shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  __syncthreads();
  if (warp == kSmallWarps) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kSmallTmem);
  }
}

struct SmallPlan {
  int splits, slabs;  // splits = 0: not a problem for this kernel
};
static int64_t small_smem_bytes(int slabs) {
  return 1024 + (int64_t)slabs * (kWBytes + kSmallTokBytes + kSmallRows * 4) + (int64_t)sizeof(SmallCtl);
}
static SmallPlan small_plan(int64_t M, int64_t N, int64_t K) {
  SmallPlan pl{0, 0};
  if (M > kSmallRows || K % kRowsBK != 0) return pl;
  const int64_t tiles = (N + kRowsBM - 1) / kRowsBM;
  if (K / kRowsBK > kSmallMaxSlabs * kMostClusterCtas || tiles > 2 * (int64_t)sm_count()) return pl;
  int most = kSmallMaxSlabs;
  while (small_smem_bytes(most) > kSmallSmem) --most;
  const int kb = (int)(K / kRowsBK);
  pl.splits = small_splits(tiles, kb, most, cluster_fits());
  if (pl.splits > 0) pl.slabs = (kb + pl.splits - 1) / pl.splits;
  return pl;
}

template <typename T>
static int launch_small(const CUtensorMap& mw, const void* x, int64_t K, const SmallPlan& pl, const RowsParams& p, cudaStream_t st) {
  auto kern = fp8_small_linear_kernel<T>;
  static thread_local bool attr_set[64] = {false};  // the opt-ins are per function and per device
  int dev = 0;
  SGLB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    SGLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.tiles_n * pl.splits), 1, 1);
  cfg.blockDim = dim3(kSmallThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)small_smem_bytes(pl.slabs);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)pl.splits, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SGLB_CUDA(cudaLaunchKernelEx(&cfg, kern, mw, static_cast<const T*>(x), K, pl.slabs, p));
  return SGLB200_OK;
}

bool small_linear_fits(int64_t M, int64_t N, int64_t K) { return small_plan(M, N, K).splits > 0; }

int small_linear(const void* x, int dtype, const void* B, const float* b_s, void* C, const void* bias, int64_t M, int64_t N,
                 int64_t K, cudaStream_t st) {
  CUtensorMap mw;
  const int rc = get_tensor_map(B, (uint64_t)K, (uint64_t)N, 1, kRowsBM, 3, &mw);
  if (rc) return rc;
  const SmallPlan pl = small_plan(M, N, K);
  RowsParams p{};
  p.b_s = b_s, p.C = C, p.bias = bias, p.M = M, p.N = N;
  p.kb_total = (int)(K / kRowsBK), p.nb_total = (int)((N + 127) / 128), p.tiles_n = p.nb_total;
  p.splits = pl.splits, p.out_fp16 = dtype;
  p.per_row = (uint32_t)((65536 + M - 1) / M);
  p.wait_probes = g_gemm_wait_probes;
  return dtype == 0 ? launch_small<__nv_bfloat16>(mw, x, K, pl, p, st) : launch_small<__half>(mw, x, K, pl, p, st);
}

int small_linear_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_small_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int small_linear_status_clear() {
  const int zero = 0;
  SGLB_CUDA(cudaMemcpyToSymbol(g_small_status, &zero, sizeof(int)));
  return SGLB200_OK;
}

}  // namespace sglb200
