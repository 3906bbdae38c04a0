// df64 instantiation of the transform kernels (kernels_impl.cuh): f64
// arithmetic on df64 words.
#include "kernels_impl.cuh"
#include "regfft.cuh"

namespace b2f {
template cudaError_t launch_lines_t<double, df>(const LinesParams&, unsigned, unsigned, size_t,
                                              cudaStream_t);
template cudaError_t launch_rader_t<double, df>(const RaderParams&, unsigned, unsigned, size_t,
                                              cudaStream_t);
template cudaError_t launch_bluestein_t<double, df>(const BluesteinParams&, unsigned, unsigned,
                                                  size_t, cudaStream_t);
template cudaError_t launch_scale_copy_t<double, df>(const void*, void*, uint64_t, double, bool,
                                                     uint32_t, cudaStream_t);
template cudaError_t launch_scale_copy_t<df, df>(const void*, void*, uint64_t, double, bool,
                                                 uint32_t, cudaStream_t);
template cudaError_t launch_blue_elem_t<double, df>(const BlueElemParams&, cudaStream_t);
template cudaError_t launch_pow2_t<double, 16, false, df>(const LinesParams&, unsigned, unsigned, size_t, cudaStream_t);
template cudaError_t launch_pow2_t<double, 16, true, df>(const LinesParams&, unsigned, unsigned, size_t, cudaStream_t);
}  // namespace b2f
