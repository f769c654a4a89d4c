// step_launch.cuh -- attributes and launch of the fused FP64 step's
// instantiations of one Riemann solver: every tile, reconstruction, and with
// or without the viscous terms (a separate instantiation: kernels without
// them keep their registers and shared memory).
#pragma once

#include "step_kernel.cuh"

namespace fv2d {

template <class T, int RS, bool VISC>
cudaError_t set_step_attrs_tile() {
  auto set = [](const void *fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  cudaError_t e = set((const void *)step_kernel<T, RECON_PCM, RS, VISC>, Smem<T, RECON_PCM, VISC>::BYTES);
  if (e == cudaSuccess) e = set((const void *)step_kernel<T, RECON_PLM, RS, VISC>, Smem<T, RECON_PLM, VISC>::BYTES);
  if (e == cudaSuccess) e = set((const void *)step_kernel<T, RECON_MH, RS, VISC>, Smem<T, RECON_MH, VISC>::BYTES);
  return e;
}

template <int RS>
cudaError_t set_step_attrs() {
  cudaError_t e = set_step_attrs_tile<WideTile, RS, false>();
  if (e == cudaSuccess) e = set_step_attrs_tile<WideTile, RS, true>();
  if (e == cudaSuccess) e = set_step_attrs_tile<SmallTile, RS, false>();
  if (e == cudaSuccess) e = set_step_attrs_tile<SmallTile, RS, true>();
  return e;
}

template <class T, int RECON, int RS, bool VISC>
cudaError_t launch_step_one(dim3 grid, cudaStream_t s, const CUtensorMap &t0, const CUtensorMap &t1,
                            const StepArgs &a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(T::NT);
  cfg.dynamicSmemBytes = Smem<T, RECON, VISC>::BYTES;
  cfg.stream = s;
  cudaLaunchAttribute overlap = {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &overlap;
  cfg.numAttrs = a.overlapped ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, step_kernel<T, RECON, RS, VISC>, t0, t1, a);
}

template <class T, int RS, bool VISC>
cudaError_t launch_step_recon(int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0, const CUtensorMap &t1,
                              const StepArgs &a) {
  switch (recon) {
    case RECON_PLM: return launch_step_one<T, RECON_PLM, RS, VISC>(grid, s, t0, t1, a);
    case RECON_MH: return launch_step_one<T, RECON_MH, RS, VISC>(grid, s, t0, t1, a);
    default: return launch_step_one<T, RECON_PCM, RS, VISC>(grid, s, t0, t1, a);
  }
}

template <int RS>
cudaError_t launch_step_rs(int tile, int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0,
                           const CUtensorMap &t1, const StepArgs &a) {
  if (tile == TILE_SMALL)
    return a.visc ? launch_step_recon<SmallTile, RS, true>(recon, grid, s, t0, t1, a)
                  : launch_step_recon<SmallTile, RS, false>(recon, grid, s, t0, t1, a);
  return a.visc ? launch_step_recon<WideTile, RS, true>(recon, grid, s, t0, t1, a)
                : launch_step_recon<WideTile, RS, false>(recon, grid, s, t0, t1, a);
}

}  // namespace fv2d
