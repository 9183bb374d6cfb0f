// Run-time register plans (fftgen.cuh): z pass with the divide, float.
#include "fftgen.cuh"

namespace exc {

template <>
void gen_zsolve<float>(const GenArgs<float>& a) {
  using C = cplx<float>;
  const int n = a.ps->n, P = a.ps->P, nkx = n / 2 + 1, ntx = (nkx + (1 << a.wlog) - 1) >> a.wlog;
  chain(gzsolve_kernel<float>, dim3((unsigned)(ntx * n), 1, a.nslots), GEN_THREADS, ((size_t)n << a.wlog) * sizeof(C), a.st, CHAIN_BLOCKS_FEW)(
      reinterpret_cast<C*>(a.ps->work), a.full, n, nkx, ntx, a.wlog, P, reinterpret_cast<const C*>(a.ps->twl_n),
      a.ps->invlap, a.sb);
}

template <>
cudaError_t configure_gen_zsolve<float>() {
  return cudaFuncSetAttribute(gzsolve_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM_MAX);
}

}  // namespace exc
