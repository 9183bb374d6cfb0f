// Register-resident two-level FFT passes for any line length L = N1 N2 with
// both factors at most gen_max_radix (the Poisson solver's passes of the grids
// without a compiled plan in fftreg.cuh; the CUFFT/FFTW plan of the
// reference's `poissonsolver` / `project!`, src/N.jl:202-307).
//
// The transform of a line is fftreg.cuh's: N1-point DFTs over the sub-lines
// m2, twiddles W_L^(m2 k1), one shared-memory exchange, N2-point DFTs over
// k1's row.  There the factors are template arguments and every grid is its
// own set of kernels; here one kernel holds every small DFT behind a switch on
// the factor, so all 17-smooth grids share five kernels.  Against the Stockham
// passes of fft.cuh (a shared-memory round trip and two barriers per radix)
// a line makes one round trip.  Projection, Stockham against these: FP32 50^3 64
// / 38 us, 90^3 77 / 54, 170^3 316 / 148, 250^3 501 / 393, 500^3 3.90 / 2.87 ms;
// FP64 20^3 96 / 46 us, 30^3 109 / 54, 50^3 197 / 101, 60^3 212 / 114; no size
// measured slower.  The switch costs registers (128, the largest DFT's), so
// two CTAs per SM: a compiled plan of the same size is a quarter faster.
#pragma once
#include <type_traits>

#include "fftmixops.cuh"
#include "fftreg.cuh"

namespace exc {

template <typename T> __host__ __device__ constexpr int gen_max_radix() { return sizeof(T) == 4 ? 34 : 17; }
constexpr int GEN_THREADS = 256;

// f(integral_constant<R>) for the run-time factor r (17-smooth, uniform over
// the block).
template <typename T, typename F>
__device__ __forceinline__ void gen_dispatch(int r, F f) {
  switch (r) {
#define EXC_R(R)                                                                       \
  case R:                                                                              \
    if constexpr (R <= gen_max_radix<T>()) f(std::integral_constant<int, R>());        \
    break;
    EXC_R(1) EXC_R(2) EXC_R(3) EXC_R(4) EXC_R(5) EXC_R(6) EXC_R(7) EXC_R(8) EXC_R(9) EXC_R(10) EXC_R(11) EXC_R(12)
    EXC_R(13) EXC_R(14) EXC_R(15) EXC_R(16) EXC_R(17) EXC_R(18) EXC_R(20) EXC_R(21) EXC_R(22) EXC_R(24) EXC_R(25)
    EXC_R(26) EXC_R(27) EXC_R(28) EXC_R(30) EXC_R(32) EXC_R(33) EXC_R(34)
#undef EXC_R
    default: break;
  }
}

// Level A of one sub-line: R values from load(m1), DFT, twiddles, to xs[k1 * step].
template <int R, bool INV, typename C, typename Load>
__device__ __forceinline__ void gen_level_a(C* xs, int step, const C* __restrict__ tl, int n2, int m2, Load load) {
  C v[R];
#pragma unroll
  for (int m1 = 0; m1 < R; ++m1) v[m1] = load(m1);
  dft_reg<R, INV>(v);
#pragma unroll
  for (int k1 = 1; k1 < R; ++k1) {
    const C w = __ldg(&tl[k1 * n2 + m2]);
    v[k1] = INV ? cmulc(v[k1], w) : cmul(v[k1], w);
  }
#pragma unroll
  for (int k1 = 0; k1 < R; ++k1) xs[k1 * step] = v[k1];
}

// A line length's factors and the reciprocals (fast_recip) of the divisions
// the kernels make by them.
struct GenLine {
  int n1 = 0, n2 = 0;
  unsigned r1 = 0, r2 = 0, rL = 0, rL1 = 0;  // of n1, n2, L, L + 1
};

// x pass geometry: rw rows per CTA; an exchange row holds [k1][m2] with rows of
// n2 | 1 words (odd: conflict-free level-B reads).
__host__ __device__ __forceinline__ int gen_xs(const GenLine& l) { return l.n1 * (l.n2 | 1); }

// ---------------------------------------------------------------------------
// Column passes: a tile is W = 2^wlog consecutive kx columns of one outer
// index; blockIdx.x = outer * ntx + tile column, blockIdx.z = slot.
// ---------------------------------------------------------------------------
// Range of the mixed-precision solve.  Its transforms are FP32, its input FP64:
// the first x pass leaves the largest biased exponent of its right-hand side per
// CTA, the first y pass folds them into a shift, 0 for right-hand sides between
// 2^-60 and 2^80 (every correction then stays within the floats).  With another
// shift the two solves that follow work on residuals scaled by 2^-shift, and the
// first correction, of the unscaled input, is taken to their units.  Where it is
// small its smallest parts may have been flushed, which the next ones make up for;
// above 2^GEN_FIRST_MAX a spectrum of n^3 of them might not fit a float, and below
// the smallest float there is none: then two corrections leave the pressure
// 3e-13 off instead of 1e-15.
constexpr int GEN_FIRST_MIN = -126, GEN_FIRST_MAX = 95;
struct GenRange {
  int* top = nullptr;    // the CTAs' exponents, then the shift
  int n = 0;             // CTAs
  __device__ __forceinline__ int shift() const { return top ? top[n] : 0; }
};
__device__ __forceinline__ double gen_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ void gen_fold_range(const GenRange& rg) {
  __shared__ int most;
  if (threadIdx.x == 0) most = 0;
  __syncthreads();
  int m = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < rg.n; i += GEN_THREADS) m = max(m, rg.top[i]);
  atomicMax(&most, m);
  __syncthreads();
  // a zero or non-finite right-hand side goes through as it is
  if (threadIdx.x == 0)
    rg.top[rg.n] = most == 0 || most == 0x7ff || (most >= 1023 - 60 && most <= 1023 + 80) ? 0 : max(most - 1023, -1000);
}

template <typename T, bool INV>
__global__ void __launch_bounds__(GEN_THREADS, 2)
gcols_kernel(cplx<T>* __restrict__ g, GenLine ln, int nkx, int ntx, int wlog, long long es, long long outer_stride,
             const cplx<T>* __restrict__ tl, SlotBatch sb, GenRange rg) {
  chain_wait();
  if (!INV && sizeof(T) == 4 && rg.top && blockIdx.x == 0) gen_fold_range(rg);
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const xs = reinterpret_cast<C*>(smem_raw);
  if (sb.active && !sb.active[blockIdx.z]) return;
  g += blockIdx.z * sb.wstride;
  const int n1 = ln.n1, n2 = ln.n2, W = 1 << wlog;
  const int outer = blockIdx.x / ntx, kx0 = (blockIdx.x - outer * ntx) << wlog;
  const int lines = min(W, nkx - kx0);
  C* const base = g + outer * outer_stride + kx0;
  gen_dispatch<T>(n1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const long long step = n2 * es;
    for (int t = threadIdx.x; t < n2 << wlog; t += GEN_THREADS) {
      const int line = t & (W - 1), m2 = t >> wlog;
      const C* const p = base + m2 * es + line;
      const bool lv = line < lines;
      gen_level_a<R, INV>(xs + t, n2 << wlog, tl, n2, m2, [&](int m1) { return lv ? p[m1 * step] : mk<T>(0, 0); });
    }
  });
  __syncthreads();
  gen_dispatch<T>(n2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const long long step = n1 * es;
    for (int t = threadIdx.x; t < n1 << wlog; t += GEN_THREADS) {
      const int line = t & (W - 1), k1 = t >> wlog;
      C v[R];
#pragma unroll
      for (int m2 = 0; m2 < R; ++m2) v[m2] = xs[((k1 * R + m2) << wlog) + line];
      dft_reg<R, INV>(v);
      if (line < lines) {
        C* const q = base + k1 * es + line;
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) q[k2 * step] = v[k2];
      }
    }
  });
}

// z pass with the spectral divide (src/N.jl:281-298).  The thread of k1
// transforms its row, divides, transforms back and puts the row back where it
// read it, so one barrier separates the levels on either side.
template <typename T>
__global__ void __launch_bounds__(GEN_THREADS, 2)
gzsolve_kernel(cplx<T>* __restrict__ g, GenLine ln, int n, int nkx, int ntx, int wlog, int P,
               const cplx<T>* __restrict__ tl, const double* __restrict__ invlap, SlotBatch sb) {
  chain_wait();
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const xs = reinterpret_cast<C*>(smem_raw);
  if (sb.active && !sb.active[blockIdx.z]) return;
  g += blockIdx.z * sb.wstride;
  const int n1 = ln.n1, n2 = ln.n2, W = 1 << wlog;
  const long long es = (long long)n * P;
  const int ky = blockIdx.x / ntx, kx0 = (blockIdx.x - ky * ntx) << wlog;
  const int lines = min(W, nkx - kx0);
  C* const base = g + (long long)ky * P + kx0;
  gen_dispatch<T>(n1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const long long step = n2 * es;
    for (int t = threadIdx.x; t < n2 << wlog; t += GEN_THREADS) {
      const int line = t & (W - 1), m2 = t >> wlog;
      const C* const p = base + m2 * es + line;
      const bool lv = line < lines;
      gen_level_a<R, false>(xs + t, n2 << wlog, tl, n2, m2, [&](int m1) { return lv ? p[m1 * step] : mk<T>(0, 0); });
    }
  });
  __syncthreads();
  gen_dispatch<T>(n2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int t = threadIdx.x; t < n1 << wlog; t += GEN_THREADS) {
      const int line = t & (W - 1), k1 = t >> wlog;
      C* const x = xs + ((k1 * R) << wlog) + line;
      C v[R];
#pragma unroll
      for (int m2 = 0; m2 < R; ++m2) v[m2] = x[m2 << wlog];
      dft_reg<R, false>(v);
      if (line < lines) {
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) {
          const long long mi = invlap_index(n, k1 + n1 * k2, ky, kx0 + line);
          if constexpr (sizeof(T) == 4) {
            // float64 factor as hi + lo floats, as in rzsolve_kernel
            const float2 f = __ldg(reinterpret_cast<const float2*>(invlap) + mi);
            v[k2].x = fmaf(v[k2].x, f.x, v[k2].x * f.y);
            v[k2].y = fmaf(v[k2].y, f.x, v[k2].y * f.y);
          } else {
            const double f = __ldg(invlap + mi);
            v[k2].x *= f;
            v[k2].y *= f;
          }
        }
      }
      dft_reg<R, true>(v);
#pragma unroll
      for (int j1 = 0; j1 < R; ++j1) {
        if (j1) v[j1] = cmulc(v[j1], __ldg(&tl[k1 * R + j1]));
        x[j1 << wlog] = v[j1];
      }
    }
  });
  __syncthreads();
  gen_dispatch<T>(n1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const long long step = n2 * es;
    for (int t = threadIdx.x; t < n2 << wlog; t += GEN_THREADS) {
      const int line = t & (W - 1), j1 = t >> wlog;
      C y[R];
#pragma unroll
      for (int k = 0; k < R; ++k) y[k] = xs[k * (n2 << wlog) + t];
      dft_reg<R, true>(y);
      if (line < lines) {
        C* const q = base + j1 * es + line;
#pragma unroll
        for (int j2 = 0; j2 < R; ++j2) q[j2 * step] = y[j2];
      }
    }
  });
}

// ---------------------------------------------------------------------------
// x passes: rows as complex lines of L = n/2 (z_m = x_2m + i x_2m+1), the
// half spectrum untangled and tangled as in fftreg.cuh.  A CTA holds rw rows in
// shared memory, word m of a row at (m / n2) (n2 | 1) + m mod n2; both levels
// work in place (level A's task owns the words m2 + n2 m1, level B's the row
// k1), and the loads and stores around them are element by element, coalesced.
// ---------------------------------------------------------------------------
template <typename T, bool INV>
__device__ __forceinline__ void gen_rows_fft(cplx<T>* xs, const GenLine& ln, int rows, const cplx<T>* __restrict__ tl) {
  using C = cplx<T>;
  const int n1 = ln.n1, n2 = ln.n2, n2p = n2 | 1, XS = n1 * n2p;
  gen_dispatch<T>(n1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int t = threadIdx.x; t < rows * n2; t += GEN_THREADS) {
      const int r = (int)fast_div((unsigned)t, ln.r2), m2 = t - r * n2;
      C* const x = xs + r * XS + m2;
      gen_level_a<R, INV>(x, n2p, tl, n2, m2, [&](int m1) { return x[m1 * n2p]; });
    }
  });
  __syncthreads();
  gen_dispatch<T>(n2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int t = threadIdx.x; t < rows * n1; t += GEN_THREADS) {
      const int r = (int)fast_div((unsigned)t, ln.r1), k1 = t - r * n1;
      C* const x = xs + r * XS + k1 * n2p;
      C v[R];
#pragma unroll
      for (int m2 = 0; m2 < R; ++m2) v[m2] = x[m2];
      dft_reg<R, INV>(v);
#pragma unroll
      for (int k2 = 0; k2 < R; ++k2) x[k2] = v[k2];
    }
  });
  __syncthreads();
}

// What the forward x pass transforms.  The last three are the FP64 steps of
// the mixed-precision solve (fftmix.cuh: mr2c_kernel's modes), FP32 only.
enum GenIn { GEN_SCAL, GEN_DIV, GEN_MIX_DIV, GEN_MIX_SCAL, GEN_MIX_RES };
template <typename T>
struct GenSrc {
  int mode;
  const T* src;  // scalar field or vector field (plain solve)
  T inv_h;
  // mixed solve: FP64 input, h, the stored right-hand side or residual d, the
  // last correction q and the one before it, the partial sums (the mean of
  // the scalar right-hand side in part[0]; with `mean` the CTA's sum of q + qp
  // goes to part[blockIdx.x])
  const double* src64;
  double h, inv_h64;
  double* d;
  const float *q, *qp;
  double* part;
  int store, mean;
  GenRange range;
};

// Where the inverse x pass puts the reals: in place at pitch 2P, or
// mc2r_kernel's modes.
enum GenTo { GEN_REAL, GEN_MIX_Q, GEN_MIX_FIN };
struct GenDst {
  int mode;
  float* q;                // GEN_MIX_Q
  double* p;               // GEN_MIX_FIN: ((q1 + q2) - mean) + c at pitch 2P
  const double* mean;      // null: no mean to remove
  const float *q1, *q2;
  GenRange range;
  int first;               // GEN_MIX_Q of the first solve
};

template <typename T>
__global__ void __launch_bounds__(GEN_THREADS, 2)
gr2c_kernel(GenSrc<T> s, GenLine ln, int n, int rw, cplx<T>* __restrict__ out, int P, const cplx<T>* __restrict__ tw,
            const cplx<T>* __restrict__ tl, SlotBatch sb) {
  chain_wait();
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const xs = reinterpret_cast<C*>(smem_raw);
  if (sb.active && !sb.active[blockIdx.y]) return;
  const T* const src = s.src + blockIdx.y * sb.ustride;
  out += blockIdx.y * sb.wstride;
  const int n1 = ln.n1, n2 = ln.n2, L = n / 2, n2p = n2 | 1, XS = n1 * n2p;
  const int nn = n * n, row0 = blockIdx.x * rw;
  const int rows = min(rw, nn - row0);
  const long long N = (long long)nn * n;
  SumF32 psum;
  // two elements per thread and turn, both elements' loads before either's
  // arithmetic (with the two-word sum of the mean, RHS and FP64 projection of
  // 250^3 2.10 -> 1.95 ms, 500^3 14.9 -> 13.6; one element 1.99 and 14.0); value =
  // load's words -> the pair of the packed line
  struct Pos {
    int r, m, base, by, bz, uy, uz, xl, xr;  // row, pair, offsets of the row and its neighbours
  };
  auto sweep = [&](auto load, auto value) {
    constexpr int U = 2;
    const int total = rows * L;
    for (int t0 = threadIdx.x; t0 < total; t0 += U * GEN_THREADS) {
      Pos p[U];
      decltype(load(p[0])) w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = min(t0 + u * GEN_THREADS, total - 1);
        const int r = (int)fast_div((unsigned)t, ln.rL), m = t - r * L;
        const int row = row0 + r, z = row / n, y = row - z * n;
        const int base = row * n;
        p[u] = {r, m, base,
                base + (y == 0 ? nn - n : -n), base + (int)(z == 0 ? N - nn : -nn),
                base + (y + 1 == n ? n - nn : n), base + (int)(z + 1 == n ? nn - N : nn),
                base + (m == 0 ? n - 1 : 2 * m - 1), base + (m == L - 1 ? 0 : 2 * m + 2)};
        w[u] = load(p[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t0 + u * GEN_THREADS < total) {
          const C v = value(p[u], w[u]);
          const int m1 = (int)fast_div((unsigned)p[u].m, ln.r2);
          xs[p[u].r * XS + m1 * n2p + (p[u].m - m1 * n2)] = v;
        }
    }
  };
  auto c_at = [](const T* f, int off, int m) { return reinterpret_cast<const C*>(f + off)[m]; };
  auto f_at = [](const float* f, int off, int m) { return reinterpret_cast<const float2*>(f + off)[m]; };
  auto d_at = [](const double* f, int off, int m) { return reinterpret_cast<const double2*>(f + off)[m]; };
  // the largest biased exponent of the right-hand side (first pass)
  int top = 0;
  auto seen = [&](double2 v) {
    top = max(top, max((__double2hiint(v.x) >> 20) & 0x7ff, (__double2hiint(v.y) >> 20) & 0x7ff));
  };
  auto put_d = [&](const Pos& p, double2 v) { reinterpret_cast<double2*>(s.d + p.base)[p.m] = v; };
  if (s.mode == GEN_SCAL) {
    sweep([&](const Pos& p) { return c_at(src, p.base, p.m); }, [](const Pos&, const C& v) { return v; });
  } else if (s.mode == GEN_DIV) {
    struct W { C a, b0, b1, c0, c1; T l; };
    const T *uy = src + N, *uz = src + 2 * N;
    sweep([&](const Pos& p) {
      return W{c_at(src, p.base, p.m), c_at(uy, p.base, p.m), c_at(uy, p.by, p.m), c_at(uz, p.base, p.m), c_at(uz, p.bz, p.m),
               src[p.xl]};
    }, [&](const Pos&, const W& w) {
      C v;
      v.x = ((w.a.x - w.l) + (w.b0.x - w.b1.x) + (w.c0.x - w.c1.x)) * s.inv_h;
      v.y = ((w.a.y - w.a.x) + (w.b0.y - w.b1.y) + (w.c0.y - w.c1.y)) * s.inv_h;
      return v;
    });
  } else if constexpr (sizeof(T) == 4) {
    if (s.mode == GEN_MIX_DIV) {
      struct W { double2 a, b0, b1, c0, c1; double l; };
      const double *ux = s.src64, *uy = ux + N, *uz = uy + N;
      sweep([&](const Pos& p) {
        return W{d_at(ux, p.base, p.m), d_at(uy, p.base, p.m), d_at(uy, p.by, p.m), d_at(uz, p.base, p.m), d_at(uz, p.bz, p.m),
                 ux[p.xl]};
      }, [&](const Pos& p, const W& w) {
        double2 dv;
        dv.x = (w.a.x - w.l) + (w.b0.x - w.b1.x) + (w.c0.x - w.c1.x);
        dv.y = (w.a.y - w.a.x) + (w.b0.y - w.b1.y) + (w.c0.y - w.c1.y);
        put_d(p, dv);
        seen(dv);
        return to_f32c<C>(dv.x, dv.y);
      });
    } else if (s.mode == GEN_MIX_SCAL) {
      const double dm = s.part[0];
      sweep([&](const Pos& p) { return d_at(s.src64, p.base, p.m); }, [&](const Pos& p, double2 dv) {
        dv.x = (dv.x - dm) * s.h;
        dv.y = (dv.y - dm) * s.h;
        put_d(p, dv);
        seen(dv);
        return to_f32c<C>(dv.x, dv.y);
      });
    } else {
      // with a shift the corrections are in units of 2^shift
      const int shift = s.range.shift();
      struct W { float2 qc, a, b, c, e, pa; float qxm, qxp; double2 dv; };
      auto residual = [&](auto shifted) {
        const double ih = shifted ? s.inv_h64 * gen_pow2(shift) : s.inv_h64, down = shifted ? gen_pow2(-shift) : 1.0;
        sweep([&](const Pos& p) {
          W w{f_at(s.q, p.base, p.m), f_at(s.q, p.by, p.m), f_at(s.q, p.uy, p.m), f_at(s.q, p.bz, p.m), f_at(s.q, p.uz, p.m),
              make_float2(0.0f, 0.0f), s.q[p.xl], s.q[p.xr], d_at(s.d, p.base, p.m)};
          if (s.mean) w.pa = f_at(s.qp, p.base, p.m);
          return w;
        }, [&](const Pos& p, const W& w) {
          double2 dv;
          dv.x = fma(-ih, stencil7_f32(w.qxm, w.qc.y, w.a.x, w.b.x, w.c.x, w.e.x, w.qc.x), w.dv.x);
          dv.y = fma(-ih, stencil7_f32(w.qc.x, w.qxp, w.a.y, w.b.y, w.c.y, w.e.y, w.qc.y), w.dv.y);
          if (s.store) put_d(p, dv);
          if (s.mean) {
            psum.add(w.pa.x);
            psum.add(w.qc.x);
            psum.add(w.pa.y);
            psum.add(w.qc.y);
          }
          if (shifted) {
            dv.x *= down;
            dv.y *= down;
          }
          return to_f32c<C>(dv.x, dv.y);
        });
      };
      if (shift) residual(std::true_type());
      else residual(std::false_type());
    }
  }
  __shared__ int most[GEN_THREADS / 32];
  const bool first = sizeof(T) == 4 && (s.mode == GEN_MIX_DIV || s.mode == GEN_MIX_SCAL);
  if (first) {
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) most[threadIdx.x >> 5] = top;
  }
  __syncthreads();
  if (first && threadIdx.x == 0) {
    for (int w = 1; w < GEN_THREADS / 32; ++w) top = max(top, most[w]);
    s.range.top[blockIdx.x] = top;
  }
  gen_rows_fft<T, false>(xs, ln, rows, tl);
  // Z_k is at row k mod n1, word k / n1
  auto at = [&](const C* x, int k) {
    const int k2 = (int)fast_div((unsigned)k, ln.r1);
    return x[(k - k2 * n1) * n2p + k2];
  };
  for (int t = threadIdx.x; t < rows * (L + 1); t += GEN_THREADS) {
    const int r = (int)fast_div((unsigned)t, ln.rL1), k = t - r * (L + 1);
    const C* const x = xs + r * XS;
    const C zk = at(x, k == L ? 0 : k), zc = cconj(at(x, k == 0 ? 0 : L - k));
    const C e = cadd(zk, zc), wo = cmul(csub(zk, zc), __ldg(&tw[k]));
    C X;
    X.x = (T)0.5 * (e.x + wo.y);
    X.y = (T)0.5 * (e.y - wo.x);
    out[(long long)(row0 + r) * P + k] = X;
  }
  if constexpr (sizeof(T) == 4) {
    if (s.mean) {  // fixed-order block sum
      __shared__ double red[GEN_THREADS / 32];
      double ps = psum.value();
      for (int o = 16; o > 0; o >>= 1) ps += __shfl_down_sync(0xffffffffu, ps, o);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ps;
      __syncthreads();
      if (threadIdx.x == 0) {
        double a = 0.0;
        for (int w = 0; w < GEN_THREADS / 32; ++w) a += red[w];
        s.part[blockIdx.x] = a;
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(GEN_THREADS, 2)
gc2r_kernel(cplx<T>* g, GenLine ln, int n, int rw, int P, const cplx<T>* __restrict__ tw,
            const cplx<T>* __restrict__ tl, GenDst d, SlotBatch sb) {
  chain_wait();
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const xs = reinterpret_cast<C*>(smem_raw);
  if (sb.active && !sb.active[blockIdx.y]) return;
  g += blockIdx.y * sb.wstride;
  const int n1 = ln.n1, n2 = ln.n2, L = n / 2, n2p = n2 | 1, XS = n1 * n2p;
  const int nn = n * n, row0 = blockIdx.x * rw;
  const int rows = min(rw, nn - row0);
  for (int t = threadIdx.x; t < rows * L; t += GEN_THREADS) {
    const int r = (int)fast_div((unsigned)t, ln.rL), k = t - r * L;
    const C* const x = g + (long long)(row0 + r) * P;
    const C xa = x[k], xb = cconj(x[L - k]);
    const C e = cadd(xa, xb), o = cmulc(csub(xa, xb), __ldg(&tw[k]));
    const int m1 = (int)fast_div((unsigned)k, ln.r2);
    xs[r * XS + m1 * n2p + (k - m1 * n2)] = mk<T>(e.x - o.y, e.y + o.x);
  }
  __syncthreads();
  gen_rows_fft<T, true>(xs, ln, rows, tl);
  // two elements per thread and turn, as in gr2c_kernel
  constexpr int U = 2;
  const int total = rows * L;
  auto word = [&](int t, int& m, int& row) {
    const int r = (int)fast_div((unsigned)t, ln.rL);
    m = t - r * L;
    row = row0 + r;
    const int k2 = (int)fast_div((unsigned)m, ln.r1);
    return xs[r * XS + (m - k2 * n1) * n2p + k2];
  };
  if (d.mode == GEN_REAL) {
    for (int t = threadIdx.x; t < total; t += GEN_THREADS) {
      int m, row;
      const C v = word(t, m, row);
      g[(long long)row * P + m] = v;
    }
  } else if constexpr (sizeof(T) == 4) {
    const int shift = d.range.shift();
    if (d.mode == GEN_MIX_Q) {
      const bool keep = shift >= GEN_FIRST_MIN && shift <= GEN_FIRST_MAX;
      const float unit = !d.first || !shift ? 1.0f : keep ? __int_as_float((127 - shift) << 23) : 0.0f;
      for (int t = threadIdx.x; t < total; t += GEN_THREADS) {
        int m, row;
        const C v = word(t, m, row);
        reinterpret_cast<float2*>(d.q + row * n)[m] = unit != 0.0f ? make_float2(f32_flush(v.x * unit), f32_flush(v.y * unit))
                                                                   : make_float2(0.0f, 0.0f);
      }
    } else {
      const bool rm = d.mean != nullptr;
      const double mu = rm ? *d.mean : 0.0;
      auto sum = [&](auto shifted) {
        for (int t0 = threadIdx.x; t0 < total; t0 += U * GEN_THREADS) {
          float2 b1[U], b2[U];
          C v[U];
          int m[U], row[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            v[u] = word(min(t0 + u * GEN_THREADS, total - 1), m[u], row[u]);
            b1[u] = reinterpret_cast<const float2*>(d.q1 + row[u] * n)[m[u]];
            b2[u] = reinterpret_cast<const float2*>(d.q2 + row[u] * n)[m[u]];
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (t0 + u * GEN_THREADS >= total) continue;
            double2 o;
            o.x = f32_to_f64(b1[u].x) + f32_to_f64(b2[u].x);
            o.y = f32_to_f64(b1[u].y) + f32_to_f64(b2[u].y);
            if (rm) {
              o.x -= mu;
              o.y -= mu;
            }
            o.x += f32_to_f64(v[u].x);
            o.y += f32_to_f64(v[u].y);
            if (shifted) {
              o.x *= gen_pow2(shift);
              o.y *= gen_pow2(shift);
            }
            reinterpret_cast<double2*>(d.p + row[u] * 2LL * P)[m[u]] = o;
          }
        }
      };
      if (shift) sum(std::true_type());
      else sum(std::false_type());
    }
  }
}

// ---------------------------------------------------------------------------
// Host side (fftgen.cu; the kernels are instantiated in fftgen_*.cu, so that
// they compile in parallel)
// ---------------------------------------------------------------------------
// The factors of line length L for radices up to maxr, most balanced first
// (n1 <= n2); false when there are none.
bool gen_line(int L, int maxr, GenLine* ln);
bool gen_plan(int n, int precision, GenLine* full, GenLine* half);
// Columns per tile (as a power of two) and rows per x-pass CTA: full cache
// lines and about 256 tasks a level, fewer where the grid would leave SMs idle.
int gen_wlog(int n, size_t csz, int nslots);
int gen_rows(int n, const GenLine& half, size_t csz, int nslots);
constexpr size_t GEN_SMEM_MAX = 80 * 1024;

template <typename T>
struct GenArgs {  // what every pass of one solve shares
  exc_poisson* ps;
  GenLine full, half;
  int wlog, rw, nslots;
  SlotBatch sb;
  cudaStream_t st;
  GenRange range;  // of a mixed solve's first y pass
};
// One pass each: y (INV: inverse), z with the divide, x forward, x inverse.
template <typename T, bool INV>
void gen_cols(const GenArgs<T>& a);
template <typename T>
void gen_zsolve(const GenArgs<T>& a);
template <typename T>
void gen_r2c(const GenArgs<T>& a, const GenSrc<T>& s);
template <typename T>
void gen_c2r(const GenArgs<T>& a, const GenDst& d);
// Their shared-memory opt-ins.
template <typename T>
cudaError_t configure_gen_cols();
template <typename T>
cudaError_t configure_gen_zsolve();
template <typename T>
cudaError_t configure_gen_x();

}  // namespace exc
