// Run-time register plans (fftgen.cuh): plan choice and the solves made of
// their passes.
#include <algorithm>

#include "fftgen.cuh"

namespace exc {

static bool radix_ok(int r) {
  for (int p : {2, 3, 5, 7, 11, 13, 17})
    while (r % p == 0) r /= p;
  return r == 1;
}

bool gen_line(int L, int maxr, GenLine* ln) {
  for (int n1 = 1, best = 0;; ++n1) {
    if (n1 * n1 <= L) {
      if (L % n1 == 0 && L / n1 <= maxr && radix_ok(n1) && radix_ok(L / n1)) best = n1;
      continue;
    }
    if (!best) return false;
    ln->n1 = best;
    ln->n2 = L / best;
    ln->r1 = fast_recip((unsigned)ln->n1);
    ln->r2 = fast_recip((unsigned)ln->n2);
    ln->rL = fast_recip((unsigned)L);
    ln->rL1 = fast_recip((unsigned)L + 1);
    return true;
  }
}

int gen_wlog(int n, size_t csz, int nslots) {
  const int nkx = n / 2 + 1;
  int w = csz == 8 ? (n >= 384 ? 3 : 4) : 3;
  while (w > 1 && (long long)((nkx + (1 << w) - 1) >> w) * n * nslots < 304) --w;
  return w;
}

int gen_rows(int n, const GenLine& half, size_t csz, int nslots) {
  int rw = GEN_THREADS / half.n1;
  const int cap = (int)(40 * 1024 / (gen_xs(half) * csz));
  if (rw > cap) rw = cap;
  const long long fill = (long long)n * n * nslots / 304;
  if (rw > fill) rw = (int)fill;
  return rw < 1 ? 1 : rw;
}

// FP64 plans stop below GEN_F64_END: from there the FP64 pipe bounds both
// forms and the Stockham passes can win (projection 150^3 833 us against 860,
// 160^3 900 against 843, 240^3 2.95 ms against 2.87).
constexpr int GEN_F64_END = 160;

bool gen_plan(int n, int precision, GenLine* full, GenLine* half) {
  const int maxr = precision == EXC_F32 ? gen_max_radix<float>() : gen_max_radix<double>();
  return n >= 4 && (precision == EXC_F32 || n < GEN_F64_END) && n % 2 == 0 && gen_line(n, maxr, full) && gen_line(n / 2, maxr, half);
}

bool gen_supported(int n, int precision) {
  GenLine a, b;
  return gen_plan(n, precision, &a, &b);
}

void gen_splits(int n, int precision, int* n1, int* h1) {
  GenLine a, b;
  gen_plan(n, precision, &a, &b);
  *n1 = a.n1;
  *h1 = b.n1;
}

void gen_geometry(int n, int precision, int* col_w, int* x_rows) {
  GenLine a, b;
  const size_t csz = precision == EXC_F32 ? 8 : 16;
  gen_plan(n, precision, &a, &b);
  *col_w = 1 << gen_wlog(n, csz, 1);
  *x_rows = gen_rows(n, b, csz, 1);
}

template <typename T>
static GenArgs<T> gen_args(exc_poisson* ps, cudaStream_t st, const SlotBatch& sb, int nslots) {
  GenArgs<T> a{};
  a.ps = ps;
  gen_plan(ps->n, sizeof(T) == 4 ? EXC_F32 : EXC_F64, &a.full, &a.half);
  a.wlog = gen_wlog(ps->n, sizeof(cplx<T>), nslots);
  a.rw = gen_rows(ps->n, a.half, sizeof(cplx<T>), nslots);
  a.nslots = nslots;
  a.sb = sb;
  a.st = st;
  return a;
}

template <typename T>
static cudaError_t solve(exc_poisson* ps, const T* src, bool vec, cudaStream_t st, const SlotBatch& sb, int nslots) {
  const GenArgs<T> a = gen_args<T>(ps, st, sb, nslots);
  GenSrc<T> s{};
  s.mode = vec ? GEN_DIV : GEN_SCAL;
  s.src = src;
  s.inv_h = (T)(1.0 / ps->h);
  gen_r2c<T>(a, s);
  gen_cols<T, false>(a);
  gen_zsolve<T>(a);
  gen_cols<T, true>(a);
  GenDst d{};
  d.mode = GEN_REAL;
  gen_c2r<T>(a, d);
  return cudaGetLastError();
}

cudaError_t gen_solve(exc_poisson* ps, const float* src, bool vec, cudaStream_t st, const SlotBatch& sb, int nslots) {
  return solve<float>(ps, src, vec, st, sb, nslots);
}
cudaError_t gen_solve(exc_poisson* ps, const double* src, bool vec, cudaStream_t st, const SlotBatch& sb, int nslots) {
  return solve<double>(ps, src, vec, st, sb, nslots);
}

// The mixed-precision solve (fftmix.cuh) on these passes: three FP32 solves,
// the residuals between them in FP64.
long long gen_mix_parts(int n) {
  GenLine full, half;
  gen_plan(n, EXC_F32, &full, &half);
  const int rw = gen_rows(n, half, sizeof(float2), 1);
  return ((long long)n * n + rw - 1) / rw;
}

cudaError_t gen_mix_solve(exc_poisson* ps, const double* src, bool vec, cudaStream_t st) {
  GenArgs<float> a = gen_args<float>(ps->mix, st, SlotBatch(), 1);
  const long long N = (long long)ps->n * ps->n * ps->n, parts = gen_mix_parts(ps->n);
  float *const q1 = ps->mix_q, *const q2 = ps->mix_q2;
  double* const mean = ps->mix_part + std::max(parts, (long long)MIX_SUM_CTAS);
  GenRange range;
  range.top = reinterpret_cast<int*>(mean + 1);
  range.n = (int)parts;
  auto columns = [&] {
    gen_cols<float, false>(a);
    gen_zsolve<float>(a);
    gen_cols<float, true>(a);
  };
  GenSrc<float> s{};
  s.src64 = src;
  s.h = ps->h;
  s.inv_h64 = 1.0 / ps->h;
  s.d = ps->mix_d;
  s.part = ps->mix_part;
  s.mode = vec ? GEN_MIX_DIV : GEN_MIX_SCAL;
  if (!vec) launch_mix_mean_of(src, N, ps->mix_part, st);
  s.range = a.range = range;
  gen_r2c<float>(a, s);
  columns();
  a.range = GenRange();
  GenDst d{};
  d.mode = GEN_MIX_Q;
  d.q = q1;
  d.range = range;
  d.first = 1;
  gen_c2r<float>(a, d);
  d.first = 0;
  s.mode = GEN_MIX_RES;
  s.q = q1;
  s.store = 1;
  gen_r2c<float>(a, s);
  columns();
  d.q = q2;
  gen_c2r<float>(a, d);
  s.q = q2;
  s.qp = q1;
  s.store = 0;
  s.mean = ps->mix_zero_mean;
  gen_r2c<float>(a, s);
  if (ps->mix_zero_mean) launch_mix_mean(ps->mix_part, (int)parts, 1.0 / (double)N, mean, st);
  columns();
  d.mode = GEN_MIX_FIN;
  d.p = reinterpret_cast<double*>(ps->work);
  d.mean = ps->mix_zero_mean ? mean : nullptr;
  d.q1 = q1;
  d.q2 = q2;
  gen_c2r<float>(a, d);
  return cudaGetLastError();
}

cudaError_t configure_gen() {
  cudaError_t e = configure_gen_cols<float>();
  if (e == cudaSuccess) e = configure_gen_cols<double>();
  if (e == cudaSuccess) e = configure_gen_zsolve<float>();
  if (e == cudaSuccess) e = configure_gen_zsolve<double>();
  if (e == cudaSuccess) e = configure_gen_x<float>();
  if (e == cudaSuccess) e = configure_gen_x<double>();
  return e;
}

}  // namespace exc
