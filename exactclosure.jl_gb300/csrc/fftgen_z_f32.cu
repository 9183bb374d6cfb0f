// Run-time register plans (fftgen.cuh): z pass with the divide, float.
#include "fftgenpass.cuh"

namespace exc {

template void gen_zsolve<float>(const GenArgs<float>&);

template <>
cudaError_t configure_gen_zsolve<float>() {
  return gen_opt_in(gzsolve_kernel<float>);
}

}  // namespace exc
