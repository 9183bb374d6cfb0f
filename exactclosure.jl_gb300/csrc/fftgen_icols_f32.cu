// Run-time register plans (fftgen.cuh): inverse y pass, float.
#include "fftgenpass.cuh"

namespace exc {

template void gen_cols<float, true>(const GenArgs<float>&);

cudaError_t configure_gen_icols_f32() { return gen_opt_in(gcols_kernel<float, true>); }

}  // namespace exc
