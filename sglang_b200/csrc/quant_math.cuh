// Arithmetic of the 1 x G quantizer on values in registers: group maximum, scale, codes (contract in quant.cu).
#pragma once
#include "common.cuh"

namespace sglb200 {

constexpr int kThreadElems = 32;  // elements of one group that a thread owns

// max(m, |a|, |b|) that returns NaN if any input is NaN: one group-wide test then tells whether the group
// holds a NaN or an infinity and must take the careful path.
__device__ __forceinline__ float max3_abs_nan(float m, float a, float b) {
  float r;
  asm("{\n\t.reg .f32 ta, tb;\n\t"
      "abs.f32 ta, %2;\n\tabs.f32 tb, %3;\n\t"
      "max.NaN.f32 %0, %1, ta, tb;\n\t}"
      : "=f"(r)
      : "f"(m), "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <typename T>
struct Chunk {  // a 16-byte chunk of T
  static constexpr int kElems = 16 / (int)sizeof(T);
  static constexpr int kPerThread = kThreadElems / kElems;  // chunks a thread owns per tile
};

template <typename T>
__device__ __forceinline__ void unpack_chunk(const uint4& raw, float* v);
template <>
__device__ __forceinline__ void unpack_chunk<__nv_bfloat16>(const uint4& raw, float* v) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void unpack_chunk<__half>(const uint4& raw, float* v) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void unpack_chunk<float>(const uint4& raw, float* v) {
  v[0] = __uint_as_float(raw.x), v[1] = __uint_as_float(raw.y);
  v[2] = __uint_as_float(raw.z), v[3] = __uint_as_float(raw.w);
}

// Pairs of 16-bit values in one word.  round_mul: the rounded pair (a, b) times `up`, rounded again (the product of two 16-bit
// floats is exact in float32, so a single packed multiply does); max_abs_nan: per half, NaN if either is.
template <typename T>
struct Packed2;
template <>
struct Packed2<__nv_bfloat16> {
  typedef __nv_bfloat162 Pair;
  static __device__ __forceinline__ void unpack(uint32_t w, float (&v)[2]) {
    v[0] = __uint_as_float(w << 16), v[1] = __uint_as_float(w & 0xffff0000u);
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) { return bits(__floats2bfloat162_rn(a, b)); }
  static __device__ __forceinline__ uint32_t round_mul(float a, float b, uint32_t up) {
    return bits(__hmul2(__floats2bfloat162_rn(a, b), pair(up)));
  }
  static __device__ __forceinline__ uint32_t max_abs_nan(uint32_t m, uint32_t w) {
    return bits(__hmax2_nan(pair(m), pair(w & 0x7fff7fffu)));
  }
  static __device__ __forceinline__ Pair pair(uint32_t w) { return *reinterpret_cast<const Pair*>(&w); }
  static __device__ __forceinline__ uint32_t bits(Pair h) { return *reinterpret_cast<const uint32_t*>(&h); }
};
template <>
struct Packed2<__half> {
  typedef __half2 Pair;
  static __device__ __forceinline__ void unpack(uint32_t w, float (&v)[2]) {
    const float2 f = __half22float2(pair(w));
    v[0] = f.x, v[1] = f.y;
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) { return bits(__floats2half2_rn(a, b)); }
  static __device__ __forceinline__ uint32_t round_mul(float a, float b, uint32_t up) {
    return bits(__hmul2(__floats2half2_rn(a, b), pair(up)));
  }
  static __device__ __forceinline__ uint32_t max_abs_nan(uint32_t m, uint32_t w) {
    return bits(__hmax2_nan(pair(m), pair(w & 0x7fff7fffu)));
  }
  static __device__ __forceinline__ Pair pair(uint32_t w) { return *reinterpret_cast<const Pair*>(&w); }
  static __device__ __forceinline__ uint32_t bits(Pair h) { return *reinterpret_cast<const uint32_t*>(&h); }
};

// Sign bits of the chunk's elements, one per byte (bit 7), in element order.
template <typename T>
__device__ __forceinline__ void chunk_signs(const uint4& raw, uint32_t* s) {
  if constexpr (sizeof(T) == 2) {
    s[0] = __byte_perm(raw.x, raw.y, 0x7531) & 0x80808080u;
    s[1] = __byte_perm(raw.z, raw.w, 0x7531) & 0x80808080u;
  } else {
    s[0] = __byte_perm(__byte_perm(raw.x, raw.y, 0x0073), __byte_perm(raw.z, raw.w, 0x0073), 0x5410) & 0x80808080u;
  }
}

// q0 = RN(x r), e = fma(-q0, scale, x), q = fma(e, r, q0) of two elements (packed float32: half the issue slots.  Cold
// inputs, 8192 x 18432 bf16: 83.8 us -> 79.7).
__device__ __forceinline__ void quotient2(float x0, float x1, float scale, float r, float& q0, float& q1) {
  asm("{\n\t.reg .b64 x, s, r, a, e;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 s, {%4, %4};\n\t"
      "mov.b64 r, {%5, %5};\n\t"
      "mul.rn.f32x2 a, x, r;\n\t"
      "fma.rn.f32x2 e, a, s, x;\n\t"
      "fma.rn.f32x2 a, e, r, a;\n\t"
      "mov.b64 {%0, %1}, a;\n\t}"
      : "=f"(q0), "=f"(q1)
      : "f"(x0), "f"(x1), "f"(-scale), "f"(r));
}

// Codes of one chunk when every element of the group is finite and the scale is in the range where the
// division-free quotient is exact (see quant_chunk_careful).  With the standard range no clamp is needed: a quotient can
// exceed 448 only by rounding and the conversion saturates; the sign of a zero quotient is taken from the
// input bits (it is the only case in which the computed sign can differ from the numerator's).
template <typename T, bool kStdRange, bool kPairs = true>
__device__ __forceinline__ void quant_chunk_fast(const uint4& raw, const float* v, float scale, float r, float qmin,
                                                 float qmax, uint32_t* codes) {
  constexpr int CE = Chunk<T>::kElems;
  float q[CE];
#pragma unroll
  for (int i = 0; i < CE; i += 2) {
    if (kPairs) {
      quotient2(v[i], v[i + 1], scale, r, q[i], q[i + 1]);
    } else {
#pragma unroll
      for (int j = i; j < i + 2; ++j) {
        const float q0 = __fmul_rn(v[j], r);
        q[j] = __fmaf_rn(__fmaf_rn(-q0, scale, v[j]), r, q0);
      }
    }
    if (!kStdRange) {
      q[i] = fminf(fmaxf(copysignf(q[i], v[i]), qmin), qmax);
      q[i + 1] = fminf(fmaxf(copysignf(q[i + 1], v[i + 1]), qmin), qmax);
    }
  }
#pragma unroll
  for (int i = 0; i < CE / 4; ++i) codes[i] = pack_e4m3x4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
  if (kStdRange) {
    uint32_t s[CE / 4];
    chunk_signs<T>(raw, s);
#pragma unroll
    for (int i = 0; i < CE / 4; ++i) codes[i] |= s[i];
  }
}

// Codes of one chunk by the full contract (any input, any scale).
//
// The contract is code = e4m3(min(max(RN(x / scale), qmin), qmax)) with an IEEE float32 division.  A
// div.rn.f32 costs about ten instructions per element, which makes the kernel issue-bound, so the quotient
// is formed without dividing (one step of Markstein's correction by the exact residual): with r = RN(1/scale) once per group,
//     q0 = RN(x*r);  e = fma(-q0, scale, x) (exact residual);  q = fma(e, r, q0);  q = copysign(q, x)
// equals RN(x / scale) bit for bit whenever |q| >= 2^-20 (checked exhaustively for every bf16 / fp16 input
// pair and on ~1e8 random float32 pairs by tests/exact_div_check.c); smaller quotients may differ in float32
// but encode as the same signed zero.  copysign restores the sign of a zero numerator.  Scales outside
// [1e-30, 1e36] (an infinite group maximum, or a caller-chosen eps near zero) take the IEEE division.
// Both clamps are applied: the lower one is also what turns a NaN quotient into -448, as in the reference.
template <typename T>
__device__ __forceinline__ void quant_chunk_careful(const float* v, float scale, float qmin, float qmax,
                                                    uint32_t* codes) {
  constexpr int CE = Chunk<T>::kElems;
  float q[CE];
  if (scale >= 1e-30f && scale <= 1e36f) {
    const float r = __frcp_rn(scale);
#pragma unroll
    for (int i = 0; i < CE; ++i) {
      const float q0 = __fmul_rn(v[i], r);
      const float e = __fmaf_rn(-q0, scale, v[i]);
      q[i] = copysignf(__fmaf_rn(e, r, q0), v[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < CE; ++i) q[i] = __fdiv_rn(v[i], scale);
  }
#pragma unroll
  for (int i = 0; i < CE; ++i) q[i] = fminf(fmaxf(q[i], qmin), qmax);
#pragma unroll
  for (int i = 0; i < CE / 4; ++i) codes[i] = pack_e4m3x4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
}

// Scale and codes of the group this thread shares with LPG - 1 neighbouring lanes.  v holds the thread's values
// (NCH chunks, one after the other), raw the bits they came from.  Every lane of the warp calls this together.
template <typename T, int LPG, bool kStdRange, int NCH = Chunk<T>::kPerThread>
__device__ __forceinline__ float quant_group(const uint4* raw, const float* v, float eps, float qmin, float qmax,
                                             uint32_t (*codes)[Chunk<T>::kElems / 4]) {
  constexpr int CE = Chunk<T>::kElems;
  float m = eps;
#pragma unroll
  for (int i = 0; i < NCH * CE; i += 2) m = max3_abs_nan(m, v[i], v[i + 1]);
#pragma unroll
  for (int off = LPG / 2; off >= 1; off >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, off));
  float scale = __fdiv_rn(m, qmax);
  if (m < __int_as_float(0x7f800000) && scale >= 1e-30f && scale <= 1e36f) {
    const float r = __frcp_rn(scale);
#pragma unroll
    for (int j = 0; j < NCH; ++j) quant_chunk_fast<T, kStdRange, (LPG >= 4)>(raw[j], v + j * CE, scale, r, qmin, qmax, codes[j]);
  } else {
    // a NaN or an infinity in the group, or an extreme scale: the reference's maximum ignores NaNs
    const unsigned lane = threadIdx.x & 31u;
    const unsigned gmask = (LPG == 32 ? 0xffffffffu : ((1u << LPG) - 1u)) << (lane & ~(unsigned)(LPG - 1));
    float a = eps;
#pragma unroll
    for (int i = 0; i < NCH * CE; ++i) a = fmaxf(a, fabsf(v[i]));
#pragma unroll
    for (int off = LPG / 2; off >= 1; off >>= 1) a = fmaxf(a, __shfl_xor_sync(gmask, a, off));
    scale = __fdiv_rn(a, qmax);
#pragma unroll
    for (int j = 0; j < NCH; ++j) quant_chunk_careful<T>(v + j * CE, scale, qmin, qmax, codes[j]);
  }
  return scale;
}

}  // namespace sglb200
