// Routing kernels that feed moe_align: softmax / sigmoid top-k and the grouped, biased "fused gate" of
// DeepSeek-V3.  One warp per token row, the row in registers (up to 1024 experts); nothing is written but the k weights
// and ids.  Each of the k picks is a warp arg-max (value descending, index ascending on ties): two warp-wide integer
// reductions over the lanes' own best entries (redux.sync on order-preserving bit patterns; five rounds of two shuffles
// each took three times as long), after which only the winner's lane looks for its next best.  The softmax gate keeps
// expert e in lane e % 32 (coalesced loads, sums in a fixed order); the fused gate gives every lane consecutive experts,
// so that a group's two largest scores come from the lanes' registers and a few shuffles instead of a serial walk
// through shared memory (64 x 256 scores: 12.7 us with the walk).  The picks stay in registers, their weights in shared memory,
// and both leave in one store each: written pick by pick and read back for the normalisation, with the scores loaded four bytes
// at a time and a division an expert for its group, the fused gate took 5.4 us for one row of 256 experts (3.8 so), 6.1 for 64
// (4.4), 30.5 for 16384 (24.5); the softmax gate 2.8 for one row of 128 experts, best eight (2.6), 14.6 for 16384 (14.0), which is
// short of issue slots; best 40 of 256 of 16384 rows 72.7 (75.3).
#include <cfloat>

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace sglb200 {

constexpr int kGateWarps = 8;          // rows per CTA
constexpr int kGateMaxPerLane = 32;    // experts <= 1024
constexpr float kNegInf = -INFINITY;

// Bit patterns that compare as unsigned integers like the floats they come from (-0 as +0).
__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t u = __float_as_uint(v + 0.f);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, m));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

// Picks the k best of sel[] (kPerLane registers per lane, the expert of register j being index(j), ascending in j) and writes their
// ids to out_i and what finish(weight(expert), sum of the k weights) gives to out_w, lane p the p-th pick of every 32.  Every lane asks
// for every weight, beside the next pick, which does not wait for it.  (Asked by lane p alone and added up behind the last pick, with
// the winner found by a vote and a shuffle: one row of 64, best 40 7.3 us for 5.5, 16384 rows 40.6 for 37.9.)  Pick p stays in
// registers of lane p; weights and ids leave once, together.
template <int kPerLane, class Index, class Weight, class Finish>
__device__ __forceinline__ float pick_topk(float (&sel)[kPerLane], Index index, Weight weight, int lane, int k, float* out_w,
                                           int32_t* out_i, Finish finish) {
  float best;  // this lane's best entry: value (never a NaN), expert (INT_MAX: nothing above -inf left) and register
  int best_e, best_j;
  auto look = [&]() {
    best = kNegInf, best_j = -1;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j)
      if (sel[j] > best) best = sel[j], best_j = j;  // ascending j = ascending expert within the lane: the first hit keeps the lower index
    best_e = best_j < 0 ? INT_MAX : index(best_j);
  };
  look();
  float sum = 0.f, mine_w = 0.f;
  int mine_e = 0;
  for (int first = 0; first < k; first += 32) {
    const int count = min(k - first, 32);
    for (int pick = 0; pick < count; ++pick) {
      const uint32_t key = ordered_bits(best), top = __reduce_max_sync(0xffffffffu, key);
      // (equal values in several lanes: the lowest expert)
      int e = __reduce_min_sync(0xffffffffu, key == top ? best_e : INT_MAX);
      if (e == INT_MAX) {
        e = 0;  // fewer candidates than k: every remaining value is -inf, and expert 0 with its weight is reported again
      } else if (best_e == e) {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
          if (j == best_j) sel[j] = kNegInf;
        look();
      }
      const float w = weight(e);
      sum += w;  // in the order of the picks, the same in every lane
      if (lane == pick) mine_e = e, mine_w = w;
    }
    if (k > 32 && lane < count) out_w[first + lane] = mine_w, out_i[first + lane] = mine_e;
  }
  if (k <= 32) {
    if (lane < k) out_w[lane] = finish(mine_w, sum), out_i[lane] = mine_e;
  } else {  // (the sum is known only now)
    for (int p = lane; p < k; p += 32) out_w[p] = finish(out_w[p], sum);
  }
  return sum;
}

// mode 0: softmax(x [tanh-capped] [+ bias]) ; weight = probability
// mode 1: sigmoid(x) [+ bias] for the selection; weight = (sigmoid + bias) - bias, as the reference reports it
template <typename T, int kPerLane, int kMode>
__global__ void __launch_bounds__(kGateWarps * 32)
    topk_gate_kernel(const T* __restrict__ gating, const float* __restrict__ bias, int64_t rows, int E, int k,
                     int renormalize, float softcap, float* __restrict__ out_w, int32_t* __restrict__ out_i) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kGateWarps + (threadIdx.x >> 5);
  ptx::launch_dependents();
  ptx::grid_dependency_wait();
  if (row >= rows) return;
  const T* x = gating + row * E;
  extern __shared__ float gate_smem[];  // per warp: E values
  float* kept = gate_smem + (threadIdx.x >> 5) * E;  // the row's weights, for the picks
  float sel[kPerLane];
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int e = j * 32 + lane;
    float v = kNegInf;
    if (e < E) {
      v = ElemTraits<T>::to_f32(x[e]);
      if (kMode == 0) {
        if (softcap != 0.f) v = tanhf(v / softcap) * softcap;
        if (bias != nullptr) v += bias[e];
      } else {
        v = 1.0f / (1.0f + expf(-v));
        const float b = bias != nullptr ? bias[e] : 0.f;
        v += b;
        kept[e] = v - b;
      }
    }
    sel[j] = v;
  }
  if (kMode == 0) {
    float mx = kNegInf;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) mx = fmaxf(mx, sel[j]);
    mx = warp_max(mx);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      sel[j] = (j * 32 + lane < E) ? expf(sel[j] - mx) : 0.f;
      s += sel[j];
    }
    const float inv = 1.f / warp_sum(s);
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      sel[j] = e < E ? sel[j] * inv : kNegInf;
      if (e < E) kept[e] = sel[j];
    }
  }
  __syncwarp();
  pick_topk<kPerLane>(
      sel, [&](int j) { return j * 32 + lane; }, [&](int e) { return kept[e]; }, lane, k, out_w + row * k, out_i + row * k,
      [&](float w, float sum) { return renormalize ? w * (1.f / sum) : w; });
}

// Lane `lane`'s N consecutive values of the E at `p` (0 past the end), 16 bytes at a time where they lie so.
template <typename T, int N>
__device__ __forceinline__ void load_run(const T* p, int E, int lane, float (&v)[N]) {
  constexpr int kVec = 16 / (int)sizeof(T);
  p += lane * N;
  if (N % kVec == 0 && E % N == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
    uint4 raw[N % kVec == 0 ? N / kVec : 1];
    const bool on = lane * N < E;
#pragma unroll
    for (int c = 0; c < N / kVec; ++c) raw[c] = on ? __ldg(reinterpret_cast<const uint4*>(p) + c) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = ElemTraits<T>::to_f32(reinterpret_cast<const T*>(raw)[j]);
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = lane * N + j < E ? ElemTraits<T>::to_f32(p[j]) : 0.f;
  }
}

// DeepSeek-V3 gate.  All arithmetic on the scores happens in the input type T, as in the reference:
//   s = T(sigmoid_f32(x)); b = s + bias (T); group score = sum of the group's two largest b (T);
//   keep the topk_group groups with the largest score (lower group index on ties); pick the top-k b among the
//   kept groups (lower expert index on ties); weights = s, divided by their sum, optionally times the scaling
//   factor.  Fused shared experts take ids E, E+1, .. and weight sum / factor before the normalisation.
// Lane l holds experts l * kPerLane .. + kPerLane - 1.
template <typename T, int kPerLane>
__global__ void __launch_bounds__(kGateWarps * 32)
    fused_gate_kernel(const T* __restrict__ input, const T* __restrict__ bias, int64_t rows, int E, int G, int topk_group,
                      int topk, int n_shared, float factor, int scale_output, float* __restrict__ out_w,
                      int32_t* __restrict__ out_i) {
  extern __shared__ float gate_smem[];  // per warp: E scores
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* score = gate_smem + warp * E;
  const int64_t row = (int64_t)blockIdx.x * kGateWarps + warp;
  ptx::launch_dependents();
  ptx::grid_dependency_wait();
  if (row >= rows) return;
  const T* x = input + row * E;
  auto biased = [](float s, float b) { return ElemTraits<T>::to_f32(ElemTraits<T>::from_f32(s + b)); };
  float sel[kPerLane], in[kPerLane], add[kPerLane];
  load_run<T, kPerLane>(x, E, lane, in);
  load_run<T, kPerLane>(bias, E, lane, add);
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int e = lane * kPerLane + j;
    sel[j] = kNegInf;
    if (e < E) {
      const float s = ElemTraits<T>::to_f32(ElemTraits<T>::from_f32(1.0f / (1.0f + expf(-in[j]))));
      score[e] = s;
      sel[j] = biased(s, add[j]);
    }
  }
  // The two largest scores of every group, of which lane g keeps group g's sum.
  const int gs = E / G, lanes_per_group = gs / kPerLane;
  float gscore = kNegInf;
  auto push = [](float v, float& m1, float& m2) {
    if (v > m1) {
      m2 = m1;
      m1 = v;
    } else if (v > m2) {
      m2 = v;
    }
  };
  const bool runs = gs % kPerLane == 0 && (lanes_per_group & (lanes_per_group - 1)) == 0;
  if (runs) {
    // a group is a run of 2^n lanes: best two of the lane's registers, merged over the run
    float m1 = -FLT_MAX, m2 = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) push(sel[j], m1, m2);
    for (int off = 1; off < lanes_per_group; off <<= 1) {
      const float o1 = __shfl_xor_sync(0xffffffffu, m1, off), o2 = __shfl_xor_sync(0xffffffffu, m2, off);
      push(o1, m1, m2);
      push(o2, m1, m2);
    }
    const float sc = ElemTraits<T>::to_f32(ElemTraits<T>::from_f32(m1 + m2));
    gscore = __shfl_sync(0xffffffffu, sc, (lane * lanes_per_group) & 31);
    if (lane >= G) gscore = kNegInf;
  } else {
    __syncwarp();
    if (lane < G) {
      float m1 = -FLT_MAX, m2 = -FLT_MAX;
      for (int i = lane * gs; i < lane * gs + gs; ++i) push(biased(score[i], ElemTraits<T>::to_f32(bias[i])), m1, m2);
      gscore = ElemTraits<T>::to_f32(ElemTraits<T>::from_f32(m1 + m2));
    }
  }
  // a group is kept when fewer than topk_group groups beat it (larger score, or equal score and lower index)
  int beaten_by = 0;
  for (int g = 0; g < G; ++g) {
    const float og = __shfl_sync(0xffffffffu, gscore, g);
    if (og > gscore || (og == gscore && g < lane)) ++beaten_by;
  }
  const uint32_t keep_mask = __ballot_sync(0xffffffffu, lane < G && beaten_by < topk_group);
  if (runs) {  // (a lane's experts are of one group)
    if (!((keep_mask >> (lane >> (__ffs(lanes_per_group) - 1))) & 1u))
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) sel[j] = kNegInf;
  } else {
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = lane * kPerLane + j;
      if (e < E && !((keep_mask >> (e / gs)) & 1u)) sel[j] = kNegInf;
    }
  }
  const int k_routed = topk - n_shared;
  float* ow = out_w + row * topk;
  int32_t* oi = out_i + row * topk;
  __syncwarp();
  auto finish = [&](float w, float sum) { return scale_output ? w / sum * factor : w / sum; };
  const float sum = pick_topk<kPerLane>(sel, [&](int j) { return lane * kPerLane + j; }, [&](int e) { return score[e]; }, lane,
                                        k_routed, ow, oi, finish);
  for (int i = lane; i < n_shared; i += 32) {
    oi[k_routed + i] = E + i;
    ow[k_routed + i] = finish(sum / factor, sum);
  }
}

template <typename T, int kMode>
static int launch_topk(const void* gating, const float* bias, int64_t rows, int E, int k, int renorm, float softcap,
                       float* out_w, int32_t* out_i, cudaStream_t st) {
  const unsigned grid = (unsigned)((rows + kGateWarps - 1) / kGateWarps);
  const T* g = static_cast<const T*>(gating);
#define SGLB_GATE_CASE(P)                                                                                        \
  if (E <= 32 * P) {                                                                                             \
    SGLB_CUDA(launch_pdl(topk_gate_kernel<T, P, kMode>, grid, kGateWarps * 32, (size_t)kGateWarps * E * sizeof(float), st, g, bias, rows, E, k, renorm, softcap, \
                         out_w, out_i));                                                                         \
    return SGLB200_OK;                                                                                           \
  }
  SGLB_GATE_CASE(1) SGLB_GATE_CASE(2) SGLB_GATE_CASE(4) SGLB_GATE_CASE(8) SGLB_GATE_CASE(16) SGLB_GATE_CASE(32)
#undef SGLB_GATE_CASE
  return fail(SGLB200_E_UNSUPPORTED, "top-k gate: %d experts (at most %d)", E, 32 * kGateMaxPerLane);
}

template <typename T>
static int launch_fused_gate(const void* input, const void* bias, int64_t rows, int E, int G, int topk_group, int topk,
                             int n_shared, float factor, int scale_output, float* out_w, int32_t* out_i,
                             cudaStream_t st) {
  const unsigned grid = (unsigned)((rows + kGateWarps - 1) / kGateWarps);
  const size_t smem = (size_t)kGateWarps * E * sizeof(float);
  const T* x = static_cast<const T*>(input);
  const T* b = static_cast<const T*>(bias);
#define SGLB_GATE_CASE(P)                                                                                      \
  if (E <= 32 * P) {                                                                                           \
    SGLB_CUDA(launch_pdl(fused_gate_kernel<T, P>, grid, kGateWarps * 32, smem, st, x, b, rows, E, G, topk_group, topk, \
                         n_shared, factor, scale_output, out_w, out_i));                                       \
    return SGLB200_OK;                                                                                         \
  }
  SGLB_GATE_CASE(1) SGLB_GATE_CASE(2) SGLB_GATE_CASE(4) SGLB_GATE_CASE(8) SGLB_GATE_CASE(16) SGLB_GATE_CASE(32)
#undef SGLB_GATE_CASE
  return fail(SGLB200_E_UNSUPPORTED, "fused gate: %d experts (at most %d)", E, 32 * kGateMaxPerLane);
}

}  // namespace sglb200

using namespace sglb200;

static int check_gate_args(const char* what, const void* gating, int dtype, int64_t rows, int E, int topk,
                           const float* out_w, const int32_t* out_i) {
  SGLB_REQUIRE(rows >= 0 && E >= 1 && topk >= 1 && topk <= E, "%s: rows=%lld experts=%d topk=%d", what, (long long)rows,
               E, topk);
  SGLB_REQUIRE(dtype >= 0 && dtype <= 2, "%s: dtype %d (0 bf16, 1 fp16, 2 fp32)", what, dtype);
  SGLB_REQUIRE(rows == 0 || (gating && out_w && out_i), "%s: null pointer", what);
  return SGLB200_OK;
}

extern "C" int sglb200_topk_softmax(const void* gating, int dtype, int64_t rows, int num_experts, int topk,
                                    int renormalize, float moe_softcapping, const float* correction_bias,
                                    float* topk_weights, int32_t* topk_ids, void* stream) {
  int rc = check_gate_args("topk_softmax", gating, dtype, rows, num_experts, topk, topk_weights, topk_ids);
  if (rc || rows == 0) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return launch_topk<__nv_bfloat16, 0>(gating, correction_bias, rows, num_experts, topk, renormalize, moe_softcapping,
                                         topk_weights, topk_ids, st);
  if (dtype == 1)
    return launch_topk<__half, 0>(gating, correction_bias, rows, num_experts, topk, renormalize, moe_softcapping,
                                  topk_weights, topk_ids, st);
  return launch_topk<float, 0>(gating, correction_bias, rows, num_experts, topk, renormalize, moe_softcapping,
                               topk_weights, topk_ids, st);
}

extern "C" int sglb200_topk_sigmoid(const void* gating, int dtype, int64_t rows, int num_experts, int topk,
                                    int renormalize, const float* correction_bias, float* topk_weights,
                                    int32_t* topk_ids, void* stream) {
  int rc = check_gate_args("topk_sigmoid", gating, dtype, rows, num_experts, topk, topk_weights, topk_ids);
  if (rc || rows == 0) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return launch_topk<__nv_bfloat16, 1>(gating, correction_bias, rows, num_experts, topk, renormalize, 0.f, topk_weights,
                                         topk_ids, st);
  if (dtype == 1)
    return launch_topk<__half, 1>(gating, correction_bias, rows, num_experts, topk, renormalize, 0.f, topk_weights,
                                  topk_ids, st);
  return launch_topk<float, 1>(gating, correction_bias, rows, num_experts, topk, renormalize, 0.f, topk_weights, topk_ids,
                               st);
}

extern "C" int sglb200_moe_fused_gate(const void* input, const void* bias, int dtype, int64_t rows, int num_experts,
                                      int num_expert_group, int topk_group, int topk, int num_fused_shared_experts,
                                      float routed_scaling_factor, int apply_routed_scaling_factor_on_output,
                                      float* topk_weights, int32_t* topk_ids, void* stream) {
  int rc = check_gate_args("moe_fused_gate", input, dtype, rows, num_experts, topk, topk_weights, topk_ids);
  if (rc) return rc;
  SGLB_REQUIRE(num_expert_group >= 1 && num_expert_group <= 32 && num_experts % num_expert_group == 0,
               "moe_fused_gate: %d groups for %d experts (1..32 groups of equal size)", num_expert_group, num_experts);
  SGLB_REQUIRE(topk_group >= 1 && topk_group <= num_expert_group, "moe_fused_gate: topk_group %d of %d groups",
               topk_group, num_expert_group);
  SGLB_REQUIRE(num_fused_shared_experts >= 0 && num_fused_shared_experts < topk,
               "moe_fused_gate: %d fused shared experts with topk %d", num_fused_shared_experts, topk);
  SGLB_REQUIRE(topk - num_fused_shared_experts <= topk_group * (num_experts / num_expert_group),
               "moe_fused_gate: topk %d exceeds the experts of %d kept groups", topk, topk_group);
  SGLB_REQUIRE(num_fused_shared_experts == 0 || routed_scaling_factor != 0.f,
               "moe_fused_gate: fused shared experts need a non-zero routed_scaling_factor");
  if (rows == 0) return SGLB200_OK;
  SGLB_REQUIRE(bias != nullptr, "moe_fused_gate: null bias");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return launch_fused_gate<__nv_bfloat16>(input, bias, rows, num_experts, num_expert_group, topk_group, topk,
                                            num_fused_shared_experts, routed_scaling_factor,
                                            apply_routed_scaling_factor_on_output, topk_weights, topk_ids, st);
  if (dtype == 1)
    return launch_fused_gate<__half>(input, bias, rows, num_experts, num_expert_group, topk_group, topk,
                                     num_fused_shared_experts, routed_scaling_factor,
                                     apply_routed_scaling_factor_on_output, topk_weights, topk_ids, st);
  return launch_fused_gate<float>(input, bias, rows, num_experts, num_expert_group, topk_group, topk,
                                  num_fused_shared_experts, routed_scaling_factor, apply_routed_scaling_factor_on_output,
                                  topk_weights, topk_ids, st);
}
