// fft_r2c_f32.cu -- FP32 x transforms of real rows (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_r2c_rows<float, float>(const float *, cplx<float> *, const R2CArgs &, const TwPair<cplx<float>> &,
                                           cudaStream_t);
template int launch_r2c_rows<float, float4>(const float4 *, cplx<float> *, const R2CArgs &,
                                            const TwPair<cplx<float>> &, cudaStream_t);
template int launch_r2c_rows<float, double>(const double *, cplx<float> *, const R2CArgs &,
                                            const TwPair<cplx<float>> &, cudaStream_t);
}  // namespace osc
