// Run-time register plans (fftgen.cuh): forward y pass, float.
#include "fftgenpass.cuh"

namespace exc {

template void gen_cols<float, false>(const GenArgs<float>&);

cudaError_t configure_gen_icols_f32();

template <>
cudaError_t configure_gen_cols<float>() {
  const cudaError_t e = gen_opt_in(gcols_kernel<float, false>);
  return e != cudaSuccess ? e : configure_gen_icols_f32();
}

}  // namespace exc
