// fft_rows_f64.cu -- FP64 x transforms (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_r2c_rows<double, double>(const double *, cplx<double> *, const R2CArgs &,
                                             const TwPair<cplx<double>> &, cudaStream_t);
template int launch_c2r_rows<double>(const cplx<double> *, const C2RArgs &, const TwPair<cplx<double>> &,
                                     cudaStream_t);
}  // namespace osc
