// fft_zconv_f32.cu -- FP32 z pass (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_zconv<float>(const cplx<float> *, cplx<float> *, const ZConvArgs &, const TwPair<cplx<float>> &,
                                 cudaStream_t);
}  // namespace osc
