// fft_lines_f64.cu -- FP64 line transforms (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_lines<double>(const cplx<double> *, cplx<double> *, const LineArgs &, int, int, bool,
                                  const TwPair<cplx<double>> &, cudaStream_t);
}  // namespace osc
