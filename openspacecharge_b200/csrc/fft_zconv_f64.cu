// fft_zconv_f64.cu -- FP64 z pass (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_zconv<double>(const cplx<double> *, cplx<double> *, const ZConvArgs &,
                                  const TwPair<cplx<double>> &, cudaStream_t);
}  // namespace osc
