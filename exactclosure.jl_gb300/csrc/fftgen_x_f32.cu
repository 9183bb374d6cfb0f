// Run-time register plans (fftgen.cuh): x passes, float.
#include "fftgenpass.cuh"

namespace exc {

template void gen_r2c<float>(const GenArgs<float>&, const GenSrc<float>&);
template void gen_c2r<float>(const GenArgs<float>&, const GenDst&);

template <>
cudaError_t configure_gen_x<float>() {
  const cudaError_t e = gen_opt_in(gr2c_kernel<float>);
  return e != cudaSuccess ? e : gen_opt_in(gc2r_kernel<float>);
}

}  // namespace exc
