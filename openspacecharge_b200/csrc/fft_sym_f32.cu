// fft_sym_f32.cu -- FP32 even/odd line transforms of the Green build (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_sym_lines<float, float, float>(const float *, float *, const SymArgs &,
                                                   const TwPair<cplx<float>> &, bool, bool, cudaStream_t);
}  // namespace osc
