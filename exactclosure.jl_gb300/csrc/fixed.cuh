// Fixed-point products and sums on the integer pipe.
//
// GB300 retires two FP64 operations per clock and SM, but 55 widening integer
// multiply-adds (32 x 32 + 64 -> 64) and about 100 integer additions
// (measured).  A double goes to an integer of BITS bits below a power of two,
// split as h 2^LOW + l with int32 parts; products of such pairs accumulate in
// three int64 sums of weight 2^(2 LOW), 2^LOW and 1, the addition part of the
// multiply-add and no carries between them; the sum is rounded to a double
// once.  The users bound their sums below 2^63.
#pragma once
#include "exc_common.cuh"

namespace exc {

struct Fx { int h, l; };
__device__ __forceinline__ Fx operator+(Fx a, Fx b) { return {a.h + b.h, a.l + b.l}; }
__device__ __forceinline__ Fx operator-(Fx a, Fx b) { return {a.h - b.h, a.l - b.l}; }
__device__ __forceinline__ Fx operator-(Fx a) { return {-a.h, -a.l}; }
struct FxSum { long long hh, m, ll; };
__device__ __forceinline__ void fx_mac(FxSum& s, Fx a, Fx b) {
  s.hh += (long long)a.h * b.h;
  s.m += (long long)a.h * b.l;
  s.m += (long long)a.l * b.h;
  s.ll += (long long)a.l * b.l;
}

// x (|x| < 2^E) in units of 2^(E - BITS), rounded to nearest; kexp = (BITS - E)
// << 20.  On the integer pipe: the FP64 pipe's own conversion takes a full
// FP64 operation's time (measured).
template <int BITS, int LOW>
__device__ __forceinline__ Fx fx_from_double(double x, int kexp) {
  static_assert(BITS >= 53 && BITS <= 62, "the mantissa and the rounding bit fit");
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  // mantissa with BITS - 52 more bits (one of them the rounding bit); shr.b64
  // gives 0 for counts of 64 and more (small values, zero)
  constexpr int UP = BITS - 52;
  const unsigned long long m5 = ((unsigned long long)__funnelshift_l(lo, mh, UP) << 32) | (lo << UP);
  unsigned long long t;
  asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"(m5), "r"(1022 + BITS - (kexp >> 20) - e));
  const long long U = (long long)((t + 1) >> 1);
  const int h = (int)((U + (1 << (LOW - 1))) >> LOW);
  const int l = (int)(unsigned)U - (h << LOW);
  const int sg = ((int)hi >> 31) | 1;
  return {h * sg, l * sg};
}

// (hh 2^(2 LOW) + m 2^LOW + ll) in units of 2^(2 LOW) times `scale`, with ten
// more bits (and 2^-10 of scale, by its exponent field) while they fit: to
// 2^-(LOW + 10 ...) below hh's unit, or to half a unit of the double.
template <int LOW>
__device__ __forceinline__ double fx_to_double(const FxSum& s, double scale) {
  const long long mm = s.m + (s.ll >> LOW);
  const long long hi = s.hh + (mm >> LOW);
  const int low10 = ((int)mm >> (LOW - 10)) & 0x3ff;
  const bool big = (unsigned)((int)(hi >> 32) + 0x200000) >= 0x400000u;  // |hi| >= 2^53
  const long long v = big ? hi : (hi << 10) | low10;
  return (double)v * __hiloint2double(__double2hiint(scale) - (big ? 0 : 10 << 20), __double2loint(scale));
}

}  // namespace exc
