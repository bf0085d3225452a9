// fft_c2r_f32.cu -- FP32 x inverse transforms (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_c2r_rows<float>(const cplx<float> *, const C2RArgs &, const TwPair<cplx<float>> &, cudaStream_t);
}  // namespace osc
