// Run-time register plans (fftgen.cuh): x passes, double.
#include "fftgenpass.cuh"

namespace exc {

template void gen_r2c<double>(const GenArgs<double>&, const GenSrc<double>&);
template void gen_c2r<double>(const GenArgs<double>&, const GenDst&);

template <>
cudaError_t configure_gen_x<double>() {
  const cudaError_t e = gen_opt_in(gr2c_kernel<double>);
  return e != cudaSuccess ? e : gen_opt_in(gc2r_kernel<double>);
}

}  // namespace exc
