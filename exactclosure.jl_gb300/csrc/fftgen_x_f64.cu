// Run-time register plans (fftgen.cuh): x passes, double.
#include "fftgen.cuh"

namespace exc {

template <>
void gen_r2c<double>(const GenArgs<double>& a, const GenSrc<double>& s) {
  using C = cplx<double>;
  const int n = a.ps->n;
  chain(gr2c_kernel<double>, dim3((unsigned)((n * n + a.rw - 1) / a.rw), a.nslots), GEN_THREADS, (size_t)a.rw * gen_xs(a.half) * sizeof(C), a.st, CHAIN_BLOCKS_FEW)(
      s, a.half, n, a.rw, reinterpret_cast<C*>(a.ps->work), a.ps->P, reinterpret_cast<const C*>(a.ps->tw),
      reinterpret_cast<const C*>(a.ps->twl_h), a.sb);
}

template <>
void gen_c2r<double>(const GenArgs<double>& a, const GenDst& d) {
  using C = cplx<double>;
  const int n = a.ps->n;
  chain(gc2r_kernel<double>, dim3((unsigned)((n * n + a.rw - 1) / a.rw), a.nslots), GEN_THREADS, (size_t)a.rw * gen_xs(a.half) * sizeof(C), a.st, CHAIN_BLOCKS_FEW)(
      reinterpret_cast<C*>(a.ps->work), a.half, n, a.rw, a.ps->P, reinterpret_cast<const C*>(a.ps->tw),
      reinterpret_cast<const C*>(a.ps->twl_h), d, a.sb);
}

template <>
cudaError_t configure_gen_x<double>() {
  cudaError_t e = cudaFuncSetAttribute(gr2c_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM_MAX);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(gc2r_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM_MAX);
}

}  // namespace exc
