// Conversions and error-free stencil sums of the mixed-precision Poisson solve
// (fftmix.cuh, fftgen.cuh).
#pragma once
#include "exc_common.cuh"

namespace exc {

// Conversions between the FP64 fields and the FP32 transforms on the integer
// pipe (the FP64 pipe, about two operations per clock per SM on GB300, is the
// solve's bottleneck), by moving the IEEE 754 binary64/binary32 fields:
// exponent rebiased by 1023 - 127 = 896, mantissa shifted by 29 bits.
//
// FP64 -> FP32 truncates the mantissa (the refinement needs about seven
// digits from each FP32 solve, not a rounded input); magnitudes below the
// smallest normal float become a signed zero, above the largest float an
// infinity, NaN stays NaN.
__device__ __forceinline__ float f64_to_f32_trunc(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned a = hi & 0x7FFFFFFFu, sign = hi & 0x80000000u;
  const unsigned t = a - 0x38000000u;  // exponent field minus 896 (in bits 30..20)
  unsigned f = (__funnelshift_l(lo, t, 3) & 0x7FFFFFFFu) | sign;
  if (a < 0x38100000u) f = sign;  // below 2^-126 (and zero)
  if (a >= 0x47F00000u) f = sign | 0x7F800000u | ((a > 0x7FF00000u || (a == 0x7FF00000u && lo)) ? 0x400000u : 0u);
  return __uint_as_float(f);
}

// FP32 -> FP64, exact for normal numbers, zeros, infinities and NaN (float
// subnormals, below 1.2e-38, become a signed zero).
__device__ __forceinline__ double f32_to_f64(float v) {
  const unsigned b = __float_as_uint(v);
  const unsigned a = b & 0x7FFFFFFFu, sign = b & 0x80000000u;
  unsigned hi = ((a >> 3) + (a >= 0x7F800000u ? 0x70000000u : 0x38000000u)) | sign;
  unsigned lo = b << 29;
  if (a < 0x00800000u) { hi = sign; lo = 0u; }
  return __hiloint2double((int)hi, (int)lo);
}

// The FP32 value the conversion above puts into p: float subnormals become a
// signed zero, so the correction kept for the next residual is the one added.
__device__ __forceinline__ float f32_flush(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x7F800000u) ? v : __uint_as_float(b & 0x80000000u);
}

// One level of error-free extraction (ExtractScalar of Rump, Ogita and Oishi,
// "Accurate floating-point summation part I: faithful rounding", SIAM J. Sci.
// Comput. 31(1), 2008): for a power of two sigma and |t| <= sigma / 2, hi =
// fl(fl(sigma + t) - sigma) is exact (Sterbenz) and a multiple of u sigma (u =
// 2^-24), and t - hi is exact with |t - hi| <= u sigma; t becomes t - hi.
__device__ __forceinline__ float extract_hi(float sigma, float& t) {
  const float hi = __fsub_rn(__fadd_rn(sigma, t), sigma);
  t = __fsub_rn(t, hi);
  return hi;
}

// (n0 + ... + n5) - 6 c of FP32 values, rounded once to FP64.  The eight
// terms (the neighbours, -4c, -2c) have |t| <= M < 2^(E+1); with sigma1 =
// 2^(E+5) every partial sum of the extracted parts is a multiple of u sigma1
// below sigma1 (sum |t| <= 8M < sigma1 / 2), so their FP32 sum h1 is exact;
// the remainders (|t| <= u sigma1) go through a second level at sigma2 =
// 2^-19 sigma1 (exact h2, a multiple of 2^(E-38)), and the last remainders
// (|t| <= 2^(E-38)) are summed in FP32, an error below 2^(E-58).  h1 + h2
// spans 43 bits and is exact in FP64; adding the last sum rounds once.  The
// six FP64 additions this replaces err by up to about 2^(E-48).
__device__ __forceinline__ double stencil7_f32(float n0, float n1, float n2, float n3, float n4, float n5,
                                               float c) {
  float t[8] = {n0, n1, n2, n3, n4, n5, -4.0f * c, -2.0f * c};
  unsigned mb = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) mb = max(mb, __float_as_uint(t[i]) & 0x7FFFFFFFu);
  // biased exponent of the largest term (0: zero or subnormal), capped so
  // sigma1 stays finite; sigma2 at least the smallest normal float
  const unsigned e1 = min((mb >> 23) + 5u, 254u);
  const float s1 = __uint_as_float(e1 << 23);
  const float s2 = __uint_as_float((e1 > 20u ? e1 - 19u : 1u) << 23);
  float h1 = 0.0f, h2 = 0.0f, l2 = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) h1 = __fadd_rn(h1, extract_hi(s1, t[i]));
#pragma unroll
  for (int i = 0; i < 8; ++i) h2 = __fadd_rn(h2, extract_hi(s2, t[i]));
#pragma unroll
  for (int i = 0; i < 8; ++i) l2 = __fadd_rn(l2, t[i]);
  return (f32_to_f64(h1) + f32_to_f64(h2)) + f32_to_f64(l2);
}

// Sum of FP32 values in two FP32 words (Knuth's TwoSum: six operations a term
// on the FP32 pipe, where an FP64 addition takes the FP64 pipe as long as 64).
// A thread sums a few hundred values of a CTA's rows: their sum is off by some
// 2^-44 of one, the mean over all threads by less than 2^-53.
struct SumF32 {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float s = __fadd_rn(hi, x), b = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
    hi = s;
  }
  __device__ __forceinline__ double value() const { return f32_to_f64(hi) + f32_to_f64(lo); }
};

template <typename C>
__device__ __forceinline__ C to_f32c(double a, double b) {
  C r;
  r.x = f64_to_f32_trunc(a);
  r.y = f64_to_f32_trunc(b);
  return r;
}

}  // namespace exc
