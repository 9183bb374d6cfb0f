// Run-time register plans (fftgen.cuh): y passes, double.
#include "fftgenpass.cuh"

namespace exc {

template void gen_cols<double, false>(const GenArgs<double>&);
template void gen_cols<double, true>(const GenArgs<double>&);

template <>
cudaError_t configure_gen_cols<double>() {
  const cudaError_t e = gen_opt_in(gcols_kernel<double, false>);
  return e != cudaSuccess ? e : gen_opt_in(gcols_kernel<double, true>);
}

}  // namespace exc
