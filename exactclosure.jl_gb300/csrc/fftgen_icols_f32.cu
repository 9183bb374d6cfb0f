// Run-time register plans (fftgen.cuh): inverse y pass, float.
#include "fftgen.cuh"

namespace exc {

template <typename T, bool INV>
void gen_cols(const GenArgs<T>& a) {
  const int n = a.ps->n, P = a.ps->P, nkx = n / 2 + 1, ntx = (nkx + (1 << a.wlog) - 1) >> a.wlog;
  chain(gcols_kernel<T, INV>, dim3((unsigned)(ntx * n), 1, a.nslots), GEN_THREADS, ((size_t)n << a.wlog) * sizeof(cplx<T>), a.st, CHAIN_BLOCKS_FEW)(
      reinterpret_cast<cplx<T>*>(a.ps->work), a.full, nkx, ntx, a.wlog, P, (long long)n * P,
      reinterpret_cast<const cplx<T>*>(a.ps->twl_n), a.sb, a.range);
}
template void gen_cols<float, true>(const GenArgs<float>&);

cudaError_t configure_gen_icols_f32() {
  return cudaFuncSetAttribute(gcols_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM_MAX);
}

}  // namespace exc
