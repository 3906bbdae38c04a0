// Launch switch of the in-place mixed-radix kernels, instantiated once per
// precision (kernels_ip_f32.cu, kernels_ip_f64.cu).
#pragma once
#include "ipfft.cuh"

namespace b2f {

template <class S>
inline cudaError_t ip_launch_t(IpKind kind, bool col, const IpParams& prm, unsigned grid,
                               unsigned threads, size_t smem, cudaStream_t st) {
  switch (kind) {
    case IP_LINES:
      return col ? launch(k_ip_lines<S, true>, prm, grid, threads, smem, st)
                 : launch(k_ip_lines<S, false>, prm, grid, threads, smem, st);
    case IP_RADER:
      return col ? launch(k_ip_rader<S, true>, prm, grid, threads, smem, st)
                 : launch(k_ip_rader<S, false>, prm, grid, threads, smem, st);
    case IP_BLUE:
      return col ? launch(k_ip_blue<S, true>, prm, grid, threads, smem, st)
                 : launch(k_ip_blue<S, false>, prm, grid, threads, smem, st);
    case IP_R2C: return launch(k_ip_r2c<S>, prm, grid, threads, smem, st);
    case IP_C2R: return launch(k_ip_c2r<S>, prm, grid, threads, smem, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace b2f
