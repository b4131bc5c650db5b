// Whole layers as one call of the C ABI: the block-FP8 linear (quantise, multiply) and the routed experts of a MoE
// layer (quantise, sort, multiply, activate + re-quantise, multiply, sum).  One workspace holds every intermediate;
// the kernels follow one another with programmatic serialization where they can, so that the start of each overlaps
// the end of the one before.
#include <algorithm>

#include "common.cuh"
#include "gemm_common.cuh"

namespace sglb200 {

constexpr float kQuantEps = 1e-10f, kFp8Max = 448.0f;

// Parts of one workspace, each on a 256-byte boundary.
struct Carver {
  int64_t bytes = 0;
  int64_t take(int64_t n) {
    const int64_t at = bytes;
    bytes += (n + 255) & ~int64_t(255);
    return at;
  }
};

struct LinearParts {
  int64_t q, s, gemm, gemm_bytes, total;
};
static LinearParts linear_parts(int64_t M, int64_t N, int64_t K) {
  LinearParts x{};
  if (small_linear_fits(M, N, K)) return x;  // no intermediates
  Carver c;
  x.q = c.take(M * K);
  x.s = c.take(M * (K / 128) * 4);
  x.gemm_bytes = sglb200_gemm_workspace_bytes(M, N, K);
  x.gemm = c.take(x.gemm_bytes);
  x.total = c.bytes;
  return x;
}

// How the routed experts run.  `tile` = activation rows per GEMM tile, `block` = padding of an expert's rows in the
// sorted order.
struct ExpertsPlan {
  int tile, block;
  int64_t cap, rows;  // entries of the sort's output; rows that can be in use
  int64_t q, s, sorted, inv, eid, post, next, cum, sort, sort_bytes, a1, a1s, ic1, a2, a2s, ic3, total;
  bool apart;         // the activation is a launch of its own between the products (128-row tiles)
  bool direct;        // one expert per token and no factor: the second GEMM writes the result itself
};

constexpr int kRowsMaxExperts = 1024;  // experts of one call of the rows kernel

// Rows per expert (tile height of the rows kernel, 0 = the 128-row kernel).  Only the average over the experts that can
// be hit is known on the host; routing spreads around it, so a tile is taken up to an average below its height: an expert
// with more rows reads its weights once per tile.  Work follows the rows that a tile has, so a height above them costs
// nothing but depth of the operand ring: 32 against 64 rows a tile, 256 experts of 7168 x 2048, in us: 0.1 rows an
// expert 242 / 242, two 1 445 / 1 441, four 1 640 / 1 609, 24 1 935 / 1 875; 128 experts of 2048 x 768 with 0.2 rows
// 53 / 55.  From 48 on the 128-row tiles are the faster ones (64 against 128 rows a tile: 48 rows 2 573 / 2 457 and
// 175 / 206, 64 rows 3 470 / 2 550 and 241 / 210): experts above 64 rows read their weights twice.
static int experts_row_tile(int64_t numel, int64_t E) {
  if (E > kRowsMaxExperts) return 0;
  const int64_t avg = numel / std::min(numel, E);
  if (avg <= 3) return 32;
  if (avg <= 48) return 64;
  return 0;
}

// Tiles of a product with `tiles_n` of them beside one another, if the experts have equally many rows.
static int64_t expert_tiles(int64_t numel, int64_t E, int64_t tiles_n) {
  const int64_t experts = std::min(numel, E);
  return experts * ((numel / experts + 127) / 128) * tiles_n;
}

// Whether the activation runs between the products instead of in the first one's epilogue.  A tile's epilogue is one to two
// microseconds longer for it, which only many tiles a CTA hide; a launch of its own takes 2 us and what it writes and reads back
// of L2, so that of one wave only the middle goes to the epilogue: fewer tiles leave SMs without a part of the work, and of more
// some are a second wave, as experts are not equal.  Us of the layer, in the epilogue / apart (tiles as estimated here, of 148
// SMs, weights from HBM): 8 tiles 25.6 / 23.2, 16 32.9 / 29.9, 32 44.0 / 42.2, 48 35.6 / 35.9, 72 42.2 / 43.6, 88 35.1 / 36.0, 96
// 47.2 / 45.6, 104 46.0 / 44.0, 128 116.6 / 111.2 and 36.1 / 37.7, 176 84.4 / 79.6, 256 97.3 / 93.4, 512 92.0 / 89.1 and 92.8 /
// 87.8, 640 117.7 / 114.2, 704 124.3 / 123.4, 768 89.6 / 89.8, 1152 155.9 / 158.0, 8448 1337 / 1409.
static bool activation_apart(int64_t numel, int64_t E, int64_t I) {
  const int64_t tiles = expert_tiles(numel, E, I / 128), sms = sm_count();
  return tiles <= 5 * sms && !(10 * tiles >= 3 * sms && 8 * tiles <= 5 * sms);
}

static ExpertsPlan experts_plan(int64_t T, int64_t k, int64_t E, int64_t H, int64_t I, int64_t Ho, float factor) {
  ExpertsPlan p{};
  const int64_t numel = T * k;
  p.tile = experts_row_tile(numel, E);
  p.block = p.tile > 0 ? 16 : 128;
  p.cap = numel + (E + 1) * (p.block - 1);
  p.rows = (numel + std::min(numel, E + 1) * (p.block - 1) + p.block - 1) / p.block * p.block;
  p.direct = k == 1 && factor == 1.0f;
  p.sort_bytes = sglb200_moe_align_workspace_bytes(numel, (int)E + 1);
  p.apart = p.tile == 0 && activation_apart(numel, E, I);
  Carver c;
  const int64_t q = T * H, s = T * (H / 128) * 4, a2 = p.rows * I, a2s = p.rows * (I / 128) * 4;
  // (codes and scales first: behind the small parts, four tokens to eight of 128 experts of 2048 x 768 46.7 -> 47.8 us)
  if (p.tile > 0) p.q = c.take(q), p.s = c.take(s);
  p.sorted = c.take(p.cap * 4), p.eid = c.take((p.cap + p.block - 1) / p.block * 4), p.post = c.take(4), p.next = c.take(8);
  p.cum = c.take((E + 2) * 4), p.sort = c.take(p.sort_bytes);
  if (p.tile > 0) {
    p.ic1 = c.take(p.rows * 2 * I * 2);
    p.a2 = c.take(a2), p.a2s = c.take(a2s);
    if (!p.direct) p.ic3 = c.take(numel * Ho * 2);
  } else {
    // Sorted rows are more than the ids by the padding of every expert, several times as many where experts average 49 rows, so
    // what is dead makes room: the codes in token order (read by the gather alone, where there is one) for the second product's
    // rows, the first product's rows and what it stores for what the second one stores.  1600 tokens of 7168 to eight of 256
    // experts: I = 2048 1.10 GB side by side, 0.75 so; I = 256 1.01 GB, 0.66.
    p.inv = c.take(numel * 4);
    Carver first = c, second = c;
    p.q = first.take(q), p.s = first.take(s);
    p.a2 = second.take(a2), p.a2s = second.take(a2s);
    c.bytes = std::max(first.bytes, second.bytes);
    first = second = c;
    p.a1 = first.take(p.rows * H), p.a1s = first.take(p.rows * (H / 128) * 4);
    if (p.apart) p.ic1 = first.take(p.rows * 2 * I * 2);
    if (!p.direct) p.ic3 = second.take(p.rows * Ho * 2);
    c.bytes = std::max(first.bytes, second.bytes);
  }
  p.total = c.bytes;
  return p;
}

}  // namespace sglb200

using namespace sglb200;

extern "C" int64_t sglb200_block_fp8_linear_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return linear_parts(M, N, K).total;
}

extern "C" int sglb200_block_fp8_linear(const void* x, int dtype, const void* W, const float* w_s, void* C, const void* bias,
                                        int64_t M, int64_t N, int64_t K, void* workspace, int64_t workspace_bytes,
                                        void* stream) {
  SGLB_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 128 == 0, "block_fp8_linear: bad shape M=%lld N=%lld K=%lld (K a multiple of 128)",
               (long long)M, (long long)N, (long long)K);
  SGLB_REQUIRE(dtype == 0 || dtype == 1, "block_fp8_linear: dtype %d (0 bf16, 1 fp16)", dtype);
  if (M == 0) return SGLB200_OK;
  if (small_linear_fits(M, N, K)) {
    SGLB_REQUIRE(x && W && w_s && C, "block_fp8_linear: null pointer");
    SGLB_REQUIRE(N % 8 == 0 && aligned16(x) && aligned16(W) && aligned16(C),
                 "block_fp8_linear: N=%lld must be a multiple of 8, x, W and C 16-byte aligned", (long long)N);
    return small_linear(x, dtype, W, w_s, C, bias, M, N, K, static_cast<cudaStream_t>(stream));
  }
  const LinearParts lp = linear_parts(M, N, K);
  if (workspace == nullptr || !aligned16(workspace) || workspace_bytes < lp.total)
    return fail(SGLB200_E_WORKSPACE, "block_fp8_linear: workspace of %lld bytes required, got %lld", (long long)lp.total,
                (long long)workspace_bytes);
  char* base = static_cast<char*>(workspace);
  float* xs = reinterpret_cast<float*>(base + lp.s);
  const int rc = quant_fp8(x, dtype, base + lp.q, xs, M, K, 128, kQuantEps, -kFp8Max, kFp8Max, K / 128, 1, true,
                           static_cast<cudaStream_t>(stream));
  if (rc) return rc;
  return scaled_mm(base + lp.q, W, xs, w_s, C, bias, M, N, K, K / 128, 1, dtype, base + lp.gemm, lp.gemm_bytes, true,
                   static_cast<cudaStream_t>(stream));
}

extern "C" int64_t sglb200_fused_experts_workspace_bytes(int64_t tokens, int64_t topk, int num_experts, int64_t hidden,
                                                         int64_t intermediate, int64_t out_hidden, float factor) {
  if (tokens <= 0 || topk <= 0 || num_experts <= 0 || hidden <= 0 || intermediate <= 0 || out_hidden <= 0) return 0;
  return experts_plan(tokens, topk, num_experts, hidden, intermediate, out_hidden, factor).total;
}

extern "C" int sglb200_fused_experts(const void* x, int dtype, const void* w13, const float* w13_s, const void* w2,
                                     const float* w2_s, const float* topk_weights, const int32_t* topk_ids, void* out,
                                     int64_t tokens, int64_t topk, int num_experts, int64_t hidden, int64_t intermediate,
                                     int64_t out_hidden, float factor, void* workspace, int64_t workspace_bytes,
                                     void* stream) {
  const int64_t T = tokens, k = topk, E = num_experts, H = hidden, I = intermediate, Ho = out_hidden, numel = T * k;
  SGLB_REQUIRE(T >= 0 && k >= 1 && E >= 1 && H > 0 && H % 128 == 0 && I > 0 && I % 128 == 0 && Ho > 0 && Ho % 8 == 0,
               "fused_experts: tokens=%lld topk=%lld experts=%lld hidden=%lld intermediate=%lld out=%lld", (long long)T,
               (long long)k, (long long)E, (long long)H, (long long)I, (long long)Ho);
  SGLB_REQUIRE(dtype == 0 || dtype == 1, "fused_experts: dtype %d (0 bf16, 1 fp16)", dtype);
  if (T == 0) return SGLB200_OK;
  SGLB_REQUIRE(x && w13 && w13_s && w2 && w2_s && topk_weights && topk_ids && out, "fused_experts: null pointer");
  SGLB_REQUIRE(aligned16(w13) && aligned16(w2) && aligned16(out), "fused_experts: weights and out must be 16-byte aligned");
  const ExpertsPlan p = experts_plan(T, k, E, H, I, Ho, factor);
  if (workspace == nullptr || !aligned16(workspace) || workspace_bytes < p.total)
    return fail(SGLB200_E_WORKSPACE, "fused_experts: workspace of %lld bytes required, got %lld", (long long)p.total,
                (long long)workspace_bytes);
  char* base = static_cast<char*>(workspace);
  auto f = [&](int64_t at) { return reinterpret_cast<float*>(base + at); };
  auto i = [&](int64_t at) { return reinterpret_cast<int32_t*>(base + at); };
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  void* ic3 = p.direct ? out : base + p.ic3;
  const int64_t hb = H / 128, ib = I / 128;
  int rc;
  int32_t* next = i(p.next);  // counters of the two products' tiles, which the sort sets to zero
  const bool beside = align_quant_fits(x, numel, (int)E + 1), sorted_rows = p.tile == 0 && !beside;
  if (beside) {
    rc = align_quant(topk_ids, numel, (int)E + 1, p.block, i(p.sorted), i(p.eid), i(p.post), i(p.cum), x, dtype, base + p.q, f(p.s), T,
                     H, kQuantEps, kFp8Max, p.tile == 0 ? i(p.inv) : nullptr, next, st);
  } else if (sorted_rows) {
    rc = align_block_size(topk_ids, numel, (int)E + 1, p.block, i(p.sorted), i(p.eid), i(p.post), i(p.cum), 1,
                          p.sort_bytes ? base + p.sort : nullptr, p.sort_bytes, i(p.inv), next, st);
    if (rc) return rc;
    rc = quant_sorted(x, dtype, base + p.a1, f(p.a1s), i(p.inv), i(p.sorted), i(p.cum), (int)E + 1, T, (int)k, H, kQuantEps, st);
  } else {
    rc = quant_fp8(x, dtype, base + p.q, f(p.s), T, H, 128, kQuantEps, -kFp8Max, kFp8Max, hb, 1, true, st);
    if (rc) return rc;
    rc = align_block_size(topk_ids, numel, (int)E + 1, p.block, i(p.sorted), i(p.eid), i(p.post), i(p.cum), 1,
                          p.sort_bytes ? base + p.sort : nullptr, p.sort_bytes, nullptr, next, st);
  }
  if (rc) return rc;
  if (p.tile > 0) {
    // Counters where either product may have more tiles than CTAs (both then run the same code, which the second finds in the
    // instruction caches): 8 experts of 4096 x 1408, 16 tokens, counters for the second alone 44.2 us, for both 42.8.
    const bool single = rows_grouped_single(p.rows, (int)E, 2 * I, p.tile) && rows_grouped_single(p.rows, (int)E, Ho, p.tile);
    if (p.direct) SGLB_CUDA(cudaMemsetAsync(out, 0, T * Ho * 2, st));  // rows of negative ids are not written below
    rc = rows_grouped_mm(base + p.q, T, hb, f(p.s), w13, w13_s, base + p.ic1, i(p.cum), i(p.sorted), nullptr, p.rows, numel, (int)E,
                         2 * I, H, (int)k, 0, dtype, p.tile, single ? nullptr : next, true, st);
    if (rc) return rc;
    rc = silu_mul_quant_fp8(base + p.ic1, dtype, base + p.a2, f(p.a2s), p.rows, I, 128, kQuantEps, i(p.post), true, st);
    if (rc) return rc;
    rc = rows_grouped_mm(base + p.a2, p.rows, ib, f(p.a2s), w2, w2_s, ic3, i(p.cum), i(p.sorted), topk_weights, p.rows, numel,
                         (int)E, Ho, I, 0, 1, dtype, p.tile, single ? nullptr : next + 1, true, st);
  } else {
    if (!sorted_rows) {
      rc = sglb200_gather_rows_fp8(base + p.q, f(p.s), base + p.a1, f(p.a1s), i(p.sorted), i(p.post), p.rows, numel, (int)k, H, hb,
                                   stream);
      if (rc) return rc;
    }
    // Gathered rows have zeros for padding.  With a tile a CTA at most, tiles that are fetched and stored whole take fewer and larger
    // copies than their quadrants: 1024 tokens to one of 8 experts of 2048 x 1024 39.4 -> 38.6 us, of 512 x 128 23.2 -> 22.8.
    auto padding = [&](int64_t n) {
      return beside && expert_tiles(numel, E, (n + 255) / 256) <= sm_count() ? Padding::kUnread : Padding::kSkipped;
    };
    if (p.apart) {
      rc = grouped_mm_any(base + p.a1, f(p.a1s), w13, w13_s, base + p.ic1, i(p.sorted), i(p.eid), i(p.post), nullptr, p.rows, numel,
                          (int)E, 2 * I, H, 0, dtype, padding(2 * I), st);
      if (rc) return rc;
      rc = silu_mul_quant_fp8(base + p.ic1, dtype, base + p.a2, f(p.a2s), p.rows, I, 128, kQuantEps, i(p.post), true, st);
    } else {
      rc = grouped_act_mm(base + p.a1, f(p.a1s), w13, w13_s, base + p.a2, f(p.a2s), i(p.sorted), i(p.eid), i(p.post),
                          p.rows, numel, (int)E, I, H, dtype, st);
    }
    if (rc) return rc;
    rc = grouped_mm_any(base + p.a2, f(p.a2s), w2, w2_s, ic3, i(p.sorted), i(p.eid), i(p.post), topk_weights, p.rows, numel, (int)E,
                        Ho, I, p.direct, dtype, padding(Ho), st);
  }
  if (rc || p.direct) return rc;
  // (the rows kernel leaves the slots of negative ids unwritten)
  if (p.tile > 0) return sglb200_moe_sum_reduce_masked(ic3, topk_ids, out, dtype, T, k, Ho, factor, stream);
  return sum_sorted(ic3, i(p.inv), out, dtype, T, k, Ho, factor, st);
}
