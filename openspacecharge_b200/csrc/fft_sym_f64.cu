// fft_sym_f64.cu -- FP64 line transforms of the Green build (fft_kernels_impl.cuh).
#include "fft_kernels_impl.cuh"

namespace osc {
template int launch_sym_lines<double, double, double>(const double *, double *, const SymArgs &,
                                                      const TwPair<cplx<double>> &, bool, bool, cudaStream_t);
template int launch_green_zlines<float>(const double *, cplx<float> *, const ZLineArgs &,
                                        const TwPair<cplx<double>> &, cudaStream_t);
template int launch_green_zlines<double>(const double *, cplx<double> *, const ZLineArgs &,
                                         const TwPair<cplx<double>> &, cudaStream_t);
}  // namespace osc
