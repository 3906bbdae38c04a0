// df64 instances of the fixed-length power-of-two kernels: f64 arithmetic,
// df64 words read and written at the ends of the plan.
#include "pow2_fixed_launch.cuh"

namespace b2f {

cudaError_t launch_pow2_fixed_df64(int lg, bool colmajor, const LinesParams& prm, unsigned grid,
                                   unsigned threads, size_t smem, cudaStream_t st) {
  return colmajor ? fx_launch_wide<double, true, df>(lg, prm, grid, threads, smem, st)
                  : fx_launch_wide<double, false, df>(lg, prm, grid, threads, smem, st);
}

}  // namespace b2f
