// Separable filter-and-sample of the DNS quantities the LES drivers need each
// step (`lazycoarsegrain(lazyfilter(.))`, src/N.jl:592-698): the fluxes r_ij =
// sigma_ij(u) + delta_ij p with their face and volume filters
// (src/N.jl:1038-1115), the volume-filtered velocity (src/N.jl:1228-1237) and
// the fine-filtered velocity at the sample points of the classic closure
// (src/N.jl:1143-1145).
//
// The kernels of these filters are products of 1-D ones, so a target is three
// passes: along x at every fine (y, z), along y at every fine z, along z.  A
// target with T taps per axis and ratio c then costs about T (1/c + 1/c^2 +
// 1/c^3) FP64 operations per fine cell instead of T^3 / c^3 times the cost of
// evaluating the source: 17 taps at ratio 5 (the box of 5 convolved with the
// reference's Gaussian of width 2H) are 4 instead of 39 source evaluations.
// The x pass evaluates every source once per fine cell (on the FP64 pipe, two
// operations per clock per SM) and shares it between all filters of it, whose
// products go to the integer pipe; all targets of a batch go through three
// launches.
//
// One lockstep step of dnsaid_project, DNS 250^3, ratio 5, that Gaussian: 165
// -> 11.7 ms, the filters (sums over T^3 taps per LES cell before) 155 -> 4.4
// ms with an x pass of 2.8 ms in FP64 (85 operations per fine cell at the
// pipe's rate), y 0.7, z 0.3; the step is 6.5 ms now.  Without the Gaussian (5 taps) 10.7 -> 9.8 ms, ratio 3 at 240^3
// 11.0 -> 10.3, 60^3 1.50 -> 1.22.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "fixed.cuh"
#include "internal.cuh"
#include "sepfilter.cuh"

namespace exc {
namespace {

constexpr int SEP_MAX_TAPSETS = 16;  // distinct 1-D stencils of one batch
constexpr int SEP_MAX_XV = 12;       // x-filtered arrays
constexpr int SEP_MAX_YV = 32;       // xy-filtered arrays
constexpr int SEP_MAX_OUT = 32;      // targets
constexpr int SEP_ROWS = 8;          // x rows per CTA
constexpr int SEP_THREADS = 256;

// Rows of n cells and `pad` ghosts on either side that an x-pass CTA stages
// beside its static words in the default 48 KB of shared memory.
constexpr size_t SEP_STATIC = 2 * (SEP_THREADS / 32) * sizeof(unsigned);
constexpr size_t sep_row_bytes(int n, int pad) { return (size_t)(n + 2 * pad) * sizeof(double); }
constexpr int sep_rows(int n, int pad) {
  const int rows = (int)((48 * 1024 - SEP_STATIC) / sep_row_bytes(n, pad));
  return rows < 1 ? 1 : rows > SEP_ROWS ? SEP_ROWS : rows;
}
// every grid and every ghost width of MAX_TAPS taps
constexpr bool sep_rows_fit() {
  for (int n = 4; n <= 1024; ++n)
    for (int pad = 0; pad <= 2 * MAX_TAPS; ++pad)
      if (sep_rows(n, pad) * sep_row_bytes(n, pad) + SEP_STATIC > 48 * 1024) return false;
  return true;
}
static_assert(sep_rows_fit(), "an x-pass CTA fits the default shared memory");

struct XVar {
  int taps;
  double* out;
};
// Fixed-point form of the x pass: values as 57-bit integers below the CTA's
// largest, weights below their list's largest, sums of at most MAX_TAPS
// products below 2^63 (halves of 2^28: 40 x 2^57 for the two middle products).
constexpr int SX_BITS = 57, SX_LOW = 29, SX_WEAK = 7;
static_assert(2 * (long long)MAX_TAPS < (1LL << (63 - 2 * (SX_BITS - SX_LOW))), "sums fit");

struct XArgs {
  Taps1D taps[SEP_MAX_TAPSETS];
  int2 wx[SEP_MAX_TAPSETS][MAX_TAPS];  // the weights in fixed point
  int we[SEP_MAX_TAPSETS];             // their exponent
  int fixed[SEP_SOURCES];              // source of blockIdx.y: fixed-point form
  int nsrc;
  int src[SEP_SOURCES];    // source of blockIdx.y
  int first[SEP_SOURCES];  // its variants are v[first .. first + count)
  int count[SEP_SOURCES];
  XVar v[SEP_MAX_XV];
  const double* u;
  const double* p;
  int n, m, c, rows;
  int z0, planes;  // fine planes of the slab, from z0 on, periodic
  int pad;  // ghost cells on either side of a staged row
  double vh;  // visc / h
};

// sigma_ij at fine cell (x, y, z): a b / 4 - (visc / h) d with a, b the
// two-point sums of u_i along j and of u_j along i, d the sum of the two
// differences (src/N.jl:106-118; the form of flux_filter_kernel).
__device__ __forceinline__ double sep_value(const XArgs& A, int src, int x, int y, int z) {
  const int n = A.n;
  const long long nn = (long long)n * n, N = nn * n;
  const long long at = (long long)z * nn + (long long)y * n + x;
  if (src < SEP_SIGMA) return A.u[src * N + at];
  if (src == SEP_P) return A.p[at];
  const int k = src - SEP_SIGMA;
  // step of one cell along axis d from (x, y, z), periodic
  auto up = [&](int d) -> long long {
    return d == 0 ? (x + 1 == n ? 1 - n : 1) : d == 1 ? (y + 1 == n ? (long long)(1 - n) * n : n)
                                                      : (z + 1 == n ? (1 - n) * nn : nn);
  };
  auto dn = [&](int d) -> long long {
    return d == 0 ? (x == 0 ? n - 1 : -1) : d == 1 ? (y == 0 ? (long long)(n - 1) * n : -n)
                                                   : (z == 0 ? (n - 1) * nn : -nn);
  };
  if (k < 3) {
    const double* f = A.u + k * N + at;
    const double r = f[0], l = f[dn(k)];
    const double s = r + l;
    return fma(-2.0 * A.vh, r - l, 0.25 * (s * s));
  }
  const int i = k - 3, j = k == 5 ? 0 : k - 2;  // s12, s23, s31
  const double* fi = A.u + i * N + at;
  const double* fj = A.u + j * N + at;
  const double il = fi[0], ir = fi[up(j)], jl = fj[0], jr = fj[up(i)];
  return fma(-A.vh, (ir + jr) - (il + jl), 0.25 * ((ir + il) * (jr + jl)));
}

// Along x.  A CTA stages `rows` rows of one source with ghosts, then applies
// every tap list of that source: in FP64, or with the values turned into
// integers in place (each word by the thread that wrote it) and the sums on the
// integer pipe (fixed.cuh), one rounding each.  A CTA stays in FP64 with a
// non-finite value, outside the exponents the scales can hold, or where 32 words
// of a row, not all zero, are below 2^-SX_WEAK of the largest: the scale would cost
// them more than its four spare bits and three (three CTAs in a thousand of a
// velocity field's quadratic stresses, none of the velocity's).
// Fixed point pays from about three products a fine cell on (the conversion is
// some 40 integer instructions a cell): four steps of 250^3, ratio 5, Gaussian 30.5
// -> 27.0 ms, 240^3, ratio 3, Gaussian 38.2 -> 36.6; without one (5 and 3 taps)
// 22.9 / 23.3 and 31.2 / 31.6, which stay in FP64.
__global__ void __launch_bounds__(SEP_THREADS) sep_x_kernel(const __grid_constant__ XArgs A) {
  extern __shared__ double row[];
  __shared__ unsigned wmax[SEP_THREADS / 32], wmin[SEP_THREADS / 32];
  static_assert(sizeof(wmax) + sizeof(wmin) == SEP_STATIC, "counted by sep_rows");
  const int n = A.n, m = A.m, c = A.c, pitch = n + 2 * A.pad;
  const int src = A.src[blockIdx.y];
  const int r0 = blockIdx.x * A.rows;
  const int rows = min(A.rows, A.planes * n - r0);
  // largest high word of a magnitude, and the smallest of the largest ones of 32
  // words that are not all zero
  unsigned top = 0, low = 0x7fffffffu;
  for (int t0 = 0; t0 < rows * pitch; t0 += SEP_THREADS) {
    const int t = t0 + threadIdx.x;
    unsigned hi = 0;
    if (t < rows * pitch) {
      const int r = t / pitch;
      const int zs = (r0 + r) / n, y = r0 + r - zs * n;
      const int z = A.z0 + zs >= n ? A.z0 + zs - n : A.z0 + zs;
      int x = t - r * pitch - A.pad;
      while (x < 0) x += n;
      while (x >= n) x -= n;
      const double q = sep_value(A, src, x, y, z);
      row[t] = q;
      hi = (unsigned)__double2hiint(q) & 0x7fffffffu;
    }
    hi = __reduce_max_sync(0xffffffffu, hi);
    top = max(top, hi);
    if (hi) low = min(low, hi);
  }
  const int v0 = A.first[blockIdx.y], vn = A.count[blockIdx.y];
  if (A.fixed[blockIdx.y]) {
    if ((threadIdx.x & 31) == 0) {
      wmax[threadIdx.x >> 5] = top;
      wmin[threadIdx.x >> 5] = low;
    }
    __syncthreads();
    for (int w = 0; w < SEP_THREADS / 32; ++w) {
      top = max(top, wmax[w]);
      low = min(low, wmin[w]);
    }
    const int E = (int)(top >> 20) - 1022;  // |value| < 2^E
    // the factor of the sums is 2^(E - 256) at the least: a normal double
    if (E > -700 && E < 800 && (low >> 20) + SX_WEAK >= top >> 20) {
      int2* const xi = reinterpret_cast<int2*>(row);
      const int kexp = (SX_BITS - E) << 20;
      for (int t = threadIdx.x; t < rows * pitch; t += SEP_THREADS) {
        const Fx q = fx_from_double<SX_BITS, SX_LOW>(row[t], kexp);
        xi[t] = make_int2(q.h, q.l);
      }
      __syncthreads();
      for (int q = threadIdx.x; q < rows * m; q += SEP_THREADS) {
        const int r = q / m, ix = q - r * m;
        const int2* f = xi + r * pitch + A.pad + c * ix;
        for (int v = v0; v < v0 + vn; ++v) {
          const int ts = A.v[v].taps;
          const Taps1D& T = A.taps[ts];
          FxSum acc{0, 0, 0};
#pragma unroll 4
          for (int t = 0; t < T.cnt; ++t) {
            const int2 w = A.wx[ts][t], x = f[T.off[t]];
            fx_mac(acc, Fx{w.x, w.y}, Fx{x.x, x.y});
          }
          const int e = E + A.we[ts] - 2 * SX_BITS + 2 * SX_LOW;
          A.v[v].out[(long long)(r0 + r) * m + ix] = fx_to_double<SX_LOW>(acc, __hiloint2double((e + 1023) << 20, 0));
        }
      }
      return;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < rows * m; q += SEP_THREADS) {
    const int r = q / m, ix = q - r * m;
    const double* f = row + r * pitch + A.pad + c * ix;
    for (int v = v0; v < v0 + vn; ++v) {
      const Taps1D& T = A.taps[A.v[v].taps];
      double acc = 0.0;
      for (int t = 0; t < T.cnt; ++t) acc = fma(T.w[t], f[T.off[t]], acc);
      A.v[v].out[(long long)(r0 + r) * m + ix] = acc;
    }
  }
}

struct YVar {
  int taps;
  const double* in;
  double* out;
};
struct YArgs {
  Taps1D taps[SEP_MAX_TAPSETS];
  YVar v[SEP_MAX_YV];
  int n, m, c, planes;
};

// Along y: [z][y][ix] -> [z][iy][ix] for the slab's planes.  The tap offsets of the
// y pass are reduced to [0, n) on the host, so one comparison wraps them.
__global__ void __launch_bounds__(SEP_THREADS) sep_y_kernel(const __grid_constant__ YArgs A) {
  const int n = A.n, m = A.m;
  const YVar V = A.v[blockIdx.y];
  const Taps1D& T = A.taps[V.taps];
  const long long tot = (long long)A.planes * m * m;
  const IdxDiv dm(m);
  for (long long g = blockIdx.x * (long long)SEP_THREADS + threadIdx.x; g < tot; g += (long long)gridDim.x * SEP_THREADS) {
    const long long r = dm.div(g);
    const int ix = (int)(g - r * m);
    const int z = (int)dm.div(r), iy = (int)(r - (long long)z * m);
    const double* f = V.in + (long long)z * n * m + ix;
    double acc = 0.0;
    for (int t = 0; t < T.cnt; ++t) {
      const int q = A.c * iy + T.off[t], y = q >= n ? q - n : q;
      acc = fma(T.w[t], f[(long long)y * m], acc);
    }
    V.out[g] = acc;
  }
}

struct ZVar {
  int taps;
  const double* in;
  const double* in2;  // second source of the target, or null
  double* out;
};
struct ZArgs {
  Taps1D taps[SEP_MAX_TAPSETS];
  ZVar v[SEP_MAX_OUT];
  int m, c;
  int i0, count;  // coarse planes of the slab
  int wrap;       // fine planes after which the slab starts again: n where it holds them all
};

// Along z: [z][iy][ix] -> [iz][iy][ix].  Offsets from the slab's first fine plane.
__global__ void __launch_bounds__(SEP_THREADS) sep_z_kernel(const __grid_constant__ ZArgs A) {
  const int m = A.m;
  const ZVar V = A.v[blockIdx.y];
  const Taps1D& T = A.taps[V.taps];
  const int mm = m * m;
  const long long tot = (long long)mm * A.count;
  const IdxDiv dmm(mm);
  for (long long g = blockIdx.x * (long long)SEP_THREADS + threadIdx.x; g < tot; g += (long long)gridDim.x * SEP_THREADS) {
    const int iz = (int)dmm.div(g), r = (int)(g - (long long)iz * mm);
    double acc = 0.0, acc2 = 0.0;
    for (int t = 0; t < T.cnt; ++t) {
      const int q = A.c * iz + T.off[t], z = q >= A.wrap ? q - A.wrap : q;
      acc = fma(T.w[t], V.in[(long long)z * mm + r], acc);
      if (V.in2) acc2 = fma(T.w[t], V.in2[(long long)z * mm + r], acc2);
    }
    V.out[(long long)A.i0 * mm + g] = acc + acc2;
  }
}

int sep_reserve(double** p, size_t* have, size_t want) {
  if (*have >= want) return EXC_OK;
  cudaFree(*p);
  *p = nullptr;
  *have = 0;
  if (cudaMalloc(p, want * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return EXC_ERR_OOM;
  }
  *have = want;
  return EXC_OK;
}

}  // namespace

void sep_free(SepWork* w) {
  cudaFree(w->a);
  cudaFree(w->b);
  *w = SepWork();
}

int SepTaps::add(int c, bool stag, bool point, const double* fdelta, int nfd, int shift) {
  Taps1D t = build_taps(c, stag, point, fdelta, nfd);
  if (t.cnt < 0) { bad = true; return 0; }
  for (int k = 0; k < t.cnt; ++k) t.off[k] += shift;
  for (size_t i = 0; i < list.size(); ++i)
    if (list[i].cnt == t.cnt && !std::memcmp(list[i].off, t.off, t.cnt * sizeof(int)) &&
        !std::memcmp(list[i].w, t.w, t.cnt * sizeof(double)))
      return (int)i;
  list.push_back(t);
  return (int)list.size() - 1;
}

int sep_filter(SepWork* w, int n, int c, double inv_h, double visc, const SepTaps& taps,
               const std::vector<SepTarget>& targets, const double* u, const double* p, cudaStream_t st) {
  if (taps.bad) { set_last_error("filter stencil longer than MAX_TAPS"); return EXC_ERR_ARG; }
  const int m = n / c;
  // distinct (source, x taps) and (x variant, y taps) pairs
  struct XV { int src, t; };
  struct YV { int x, t; };
  std::vector<XV> xv;
  std::vector<YV> yv;
  auto xvar = [&](int src, int t) {
    for (size_t i = 0; i < xv.size(); ++i)
      if (xv[i].src == src && xv[i].t == t) return (int)i;
    xv.push_back({src, t});
    return (int)xv.size() - 1;
  };
  auto yvar = [&](int x, int t) {
    for (size_t i = 0; i < yv.size(); ++i)
      if (yv[i].x == x && yv[i].t == t) return (int)i;
    yv.push_back({x, t});
    return (int)yv.size() - 1;
  };
  std::vector<int> y1, y2;
  for (const SepTarget& T : targets) {
    y1.push_back(yvar(xvar(T.src, T.t[0]), T.t[1]));
    y2.push_back(T.src2 >= 0 ? yvar(xvar(T.src2, T.t[0]), T.t[1]) : -1);
  }
  if (taps.list.size() > SEP_MAX_TAPSETS || xv.size() > SEP_MAX_XV || yv.size() > SEP_MAX_YV ||
      targets.size() > SEP_MAX_OUT) {
    set_last_error("too many filters in one batch");
    return EXC_ERR_ARG;
  }
  // The whole grid at once while its scratch stays below SEP_SCRATCH, else slabs of
  // `count` coarse planes with the fine planes their z taps reach, down to the
  // memory there is
  int zlo = 0, zhi = 0;
  for (const SepTarget& T : targets) {
    const Taps1D& z = taps.list[T.t[2]];
    for (int k = 0; k < z.cnt; ++k) {
      zlo = std::min(zlo, z.off[k]);
      zhi = std::max(zhi, z.off[k]);
    }
  }
  const size_t plane = xv.size() * n * m + yv.size() * m * m;  // words a fine plane
  auto planes_of = [&](int count) { return c * (count - 1) + zhi - zlo + 1; };
  int count = m;
  bool whole = plane * n * sizeof(double) <= w->limit;
  while (!whole && count > 1 && plane * planes_of(count) * sizeof(double) > w->limit) count = (count + 1) / 2;
  for (;; whole = false, count = (count + 1) / 2) {
    if (planes_of(count) >= n) whole = true;
    const size_t planes = whole ? n : planes_of(count);
    if (sep_reserve(&w->a, &w->na, xv.size() * planes * n * m) == EXC_OK &&
        sep_reserve(&w->b, &w->nb, yv.size() * planes * m * m) == EXC_OK)
      break;
    cudaFree(w->a);
    cudaFree(w->b);
    w->a = w->b = nullptr;
    w->na = w->nb = 0;
    if (count == 1) { set_last_error("out of device memory (filter scratch)"); return EXC_ERR_OOM; }
  }
  const int planes = whole ? n : planes_of(count);
  if (whole) count = m;
  const size_t xw = (size_t)planes * n * m, yw = (size_t)planes * m * m;

  XArgs X{};
  YArgs Y{};
  ZArgs Z{};
  int pad = 0;
  bool ok[SEP_MAX_TAPSETS];
  for (size_t i = 0; i < taps.list.size(); ++i) {
    X.taps[i] = Y.taps[i] = taps.list[i];
    for (int k = 0; k < Y.taps[i].cnt; ++k) Y.taps[i].off[k] = ((Y.taps[i].off[k] % n) + n) % n;
    Z.taps[i] = whole ? Y.taps[i] : X.taps[i];
    for (int k = 0; !whole && k < Z.taps[i].cnt; ++k) Z.taps[i].off[k] -= zlo;
    // |w| < 2^we; weights outside the range of the scales stay in FP64
    double top = 0.0;
    for (int k = 0; k < X.taps[i].cnt; ++k) top = std::max(top, std::fabs(X.taps[i].w[k]));
    int e = 0;
    if (top > 0.0 && std::isfinite(top)) std::frexp(top, &e);
    X.we[i] = e;
    ok[i] = std::isfinite(top) && e > -200 && e < 200;
    for (int k = 0; ok[i] && k < X.taps[i].cnt; ++k) {
      const long long W = std::llrint(std::ldexp(X.taps[i].w[k], SX_BITS - e));
      const long long h = (W + (1LL << (SX_LOW - 1))) >> SX_LOW;
      X.wx[i][k] = make_int2((int)h, (int)(W - h * (1LL << SX_LOW)));
    }
  }
  X.u = u;
  X.p = p;
  X.n = Y.n = n;
  X.planes = Y.planes = planes;
  Z.wrap = whole ? n : planes;
  X.m = Y.m = Z.m = m;
  X.c = Y.c = Z.c = c;
  X.vh = visc * inv_h;
  // sources in order, the variants of one source together
  std::vector<int> slot(xv.size());
  int used = 0;
  for (int s = 0; s < SEP_SOURCES; ++s) {
    int cnt = 0, products = 0;
    bool fits = true;
    for (size_t i = 0; i < xv.size(); ++i)
      if (xv[i].src == s) {
        const Taps1D& T = taps.list[xv[i].t];
        for (int k = 0; k < T.cnt; ++k) {
          // farthest reach beyond the row: c ix + off over ix < m
          if (-T.off[k] > pad) pad = -T.off[k];
          if (T.off[k] - (c - 1) > pad) pad = T.off[k] - (c - 1);
        }
        products += T.cnt;
        fits = fits && ok[xv[i].t];
        slot[i] = used + cnt;
        X.v[used + cnt] = {xv[i].t, w->a + (size_t)(used + cnt) * xw};
        ++cnt;
      }
    if (!cnt) continue;
    X.fixed[X.nsrc] = fits && products > 3 * c;
    X.src[X.nsrc] = s;
    X.first[X.nsrc] = used;
    X.count[X.nsrc] = cnt;
    ++X.nsrc;
    used += cnt;
  }
  X.pad = pad;
  for (size_t i = 0; i < yv.size(); ++i)
    Y.v[i] = {yv[i].t, w->a + (size_t)slot[yv[i].x] * xw, w->b + i * yw};
  for (size_t i = 0; i < targets.size(); ++i)
    Z.v[i] = {targets[i].t[2], w->b + (size_t)y1[i] * yw, y2[i] >= 0 ? w->b + (size_t)y2[i] * yw : nullptr,
              targets[i].out};

  const int rows = X.rows = sep_rows(n, pad);
  auto blocks = [](size_t cnt) {
    const size_t b = (cnt + SEP_THREADS - 1) / SEP_THREADS;
    return (unsigned)(b < 152 * 16 ? b : 152 * 16);
  };
  for (int i0 = 0; i0 < m; i0 += count) {
    X.z0 = whole ? 0 : (((c * i0 + zlo) % n) + n) % n;
    Z.i0 = i0;
    Z.count = std::min(count, m - i0);
    sep_x_kernel<<<dim3((unsigned)((planes * n + rows - 1) / rows), X.nsrc), SEP_THREADS, rows * sep_row_bytes(n, pad), st>>>(X);
    sep_y_kernel<<<dim3(blocks(yw), (unsigned)yv.size()), SEP_THREADS, 0, st>>>(Y);
    sep_z_kernel<<<dim3(blocks((size_t)m * m * Z.count), (unsigned)targets.size()), SEP_THREADS, 0, st>>>(Z);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error(cudaGetErrorString(e)); return EXC_ERR_CUDA; }
  return EXC_OK;
}

}  // namespace exc
