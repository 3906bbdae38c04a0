// f64 instances of the in-place mixed-radix kernels.
#include "ip_launch.cuh"

namespace b2f {

cudaError_t launch_ip_f64(IpKind kind, bool col, const IpParams& prm, unsigned grid,
                          unsigned threads, size_t smem, cudaStream_t st) {
  return ip_launch_t<double>(kind, col, prm, grid, threads, smem, st);
}

}  // namespace b2f
