// fft_lines_f32.cu -- FP32 line transforms (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_lines<float>(const cplx<float> *, cplx<float> *, const LineArgs &, int, int, bool,
                                 const TwPair<cplx<float>> &, cudaStream_t);
}  // namespace osc
