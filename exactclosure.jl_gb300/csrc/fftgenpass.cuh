// Launchers of the run-time register plans' passes (fftgen.cuh): included by the
// fftgen_*.cu, each of which instantiates some of them.
#pragma once
#include "fftgen.cuh"

namespace exc {

template <typename K>
cudaError_t gen_opt_in(K* kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM_MAX);
}

template <typename T, bool INV>
void gen_cols(const GenArgs<T>& a) {
  using C = cplx<T>;
  const int n = a.ps->n, P = a.ps->P, nkx = n / 2 + 1, ntx = (nkx + (1 << a.wlog) - 1) >> a.wlog;
  chain(gcols_kernel<T, INV>, dim3((unsigned)(ntx * n), 1, a.nslots), GEN_THREADS, ((size_t)n << a.wlog) * sizeof(C),
        a.st, CHAIN_BLOCKS_FEW)(reinterpret_cast<C*>(a.ps->work), a.full, nkx, ntx, a.wlog, P, (long long)n * P,
                                reinterpret_cast<const C*>(a.ps->twl_n), a.sb, a.range);
}

template <typename T>
void gen_zsolve(const GenArgs<T>& a) {
  using C = cplx<T>;
  const int n = a.ps->n, P = a.ps->P, nkx = n / 2 + 1, ntx = (nkx + (1 << a.wlog) - 1) >> a.wlog;
  chain(gzsolve_kernel<T>, dim3((unsigned)(ntx * n), 1, a.nslots), GEN_THREADS, ((size_t)n << a.wlog) * sizeof(C), a.st,
        CHAIN_BLOCKS_FEW)(reinterpret_cast<C*>(a.ps->work), a.full, n, nkx, ntx, a.wlog, P,
                          reinterpret_cast<const C*>(a.ps->twl_n), a.ps->invlap, a.sb);
}

template <typename T>
void gen_r2c(const GenArgs<T>& a, const GenSrc<T>& s) {
  using C = cplx<T>;
  const int n = a.ps->n;
  chain(gr2c_kernel<T>, dim3((unsigned)((n * n + a.rw - 1) / a.rw), a.nslots), GEN_THREADS,
        (size_t)a.rw * gen_xs(a.half) * sizeof(C), a.st, CHAIN_BLOCKS_FEW)(
      s, a.half, n, a.rw, reinterpret_cast<C*>(a.ps->work), a.ps->P, reinterpret_cast<const C*>(a.ps->tw),
      reinterpret_cast<const C*>(a.ps->twl_h), a.sb);
}

template <typename T>
void gen_c2r(const GenArgs<T>& a, const GenDst& d) {
  using C = cplx<T>;
  const int n = a.ps->n;
  chain(gc2r_kernel<T>, dim3((unsigned)((n * n + a.rw - 1) / a.rw), a.nslots), GEN_THREADS,
        (size_t)a.rw * gen_xs(a.half) * sizeof(C), a.st, CHAIN_BLOCKS_FEW)(
      reinterpret_cast<C*>(a.ps->work), a.half, n, a.rw, a.ps->P, reinterpret_cast<const C*>(a.ps->tw),
      reinterpret_cast<const C*>(a.ps->twl_h), d, a.sb);
}

}  // namespace exc
