// Run-time register plans (fftgen.cuh): z pass with the divide, double.
#include "fftgenpass.cuh"

namespace exc {

template void gen_zsolve<double>(const GenArgs<double>&);

template <>
cudaError_t configure_gen_zsolve<double>() {
  return gen_opt_in(gzsolve_kernel<double>);
}

}  // namespace exc
