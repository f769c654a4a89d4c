// step_hll.cu -- instantiations of the fused FP64 step for the HLL solver
// (one translation unit per solver so that they compile in parallel).
#include "step_launch.cuh"

namespace fv2d {
cudaError_t set_step_attrs_hll() { return set_step_attrs<RS_HLL>(); }
cudaError_t launch_step_hll(int tile, int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0,
                            const CUtensorMap &t1, const StepArgs &a) {
  return launch_step_rs<RS_HLL>(tile, recon, grid, s, t0, t1, a);
}
}  // namespace fv2d
