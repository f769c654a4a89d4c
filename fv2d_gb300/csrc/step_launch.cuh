// step_launch.cuh -- attributes and launch of the fused FP64 step's
// instantiations of one Riemann solver: every tile, reconstruction and form
// (StepForm).
#pragma once

#include "step_kernel.cuh"

namespace fv2d {

// The form that stands in for one that is not compiled.
template <class T, int RECON, int RS>
constexpr int step_form(int form) {
  return form == FORM_PLAIN && !has_plain_form<T, RECON, RS>() ? (int)FORM_SOURCES : form;
}

template <class T, int RECON, int RS, int FORM>
cudaError_t set_step_attrs_one() {
  return cudaFuncSetAttribute((const void *)step_kernel<T, RECON, RS, step_form<T, RECON, RS>(FORM)>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)Smem<T, RECON, FORM == FORM_VISCOUS>::BYTES);
}

template <class T, int RS, int FORM>
cudaError_t set_step_attrs_tile() {
  cudaError_t e = set_step_attrs_one<T, RECON_PCM, RS, FORM>();
  if (e == cudaSuccess) e = set_step_attrs_one<T, RECON_PLM, RS, FORM>();
  if (e == cudaSuccess) e = set_step_attrs_one<T, RECON_MH, RS, FORM>();
  return e;
}

template <class T, int RS>
cudaError_t set_step_attrs_forms() {
  cudaError_t e = set_step_attrs_tile<T, RS, FORM_PLAIN>();
  if (e == cudaSuccess) e = set_step_attrs_tile<T, RS, FORM_SOURCES>();
  if (e == cudaSuccess) e = set_step_attrs_tile<T, RS, FORM_VISCOUS>();
  return e;
}

template <int RS>
cudaError_t set_step_attrs() {
  const cudaError_t e = set_step_attrs_forms<WideTile, RS>();
  return e == cudaSuccess ? set_step_attrs_forms<SmallTile, RS>() : e;
}

template <class T, int RECON, int RS, int FORM>
cudaError_t launch_step_one(dim3 grid, cudaStream_t s, const CUtensorMap &t0, const CUtensorMap &t1,
                            const StepArgs &a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(T::NT);
  cfg.dynamicSmemBytes = Smem<T, RECON, FORM == FORM_VISCOUS>::BYTES;
  cfg.stream = s;
  cudaLaunchAttribute overlap = {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &overlap;
  cfg.numAttrs = a.overlapped ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, step_kernel<T, RECON, RS, step_form<T, RECON, RS>(FORM)>, t0, t1, a);
}

template <class T, int RS, int FORM>
cudaError_t launch_step_recon(int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0, const CUtensorMap &t1,
                              const StepArgs &a) {
  switch (recon) {
    case RECON_PLM: return launch_step_one<T, RECON_PLM, RS, FORM>(grid, s, t0, t1, a);
    case RECON_MH: return launch_step_one<T, RECON_MH, RS, FORM>(grid, s, t0, t1, a);
    default: return launch_step_one<T, RECON_PCM, RS, FORM>(grid, s, t0, t1, a);
  }
}

template <class T, int RS>
cudaError_t launch_step_form(int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0, const CUtensorMap &t1,
                             const StepArgs &a) {
  if (a.visc) return launch_step_recon<T, RS, FORM_VISCOUS>(recon, grid, s, t0, t1, a);
  if (a.stage != STAGE_EULER || a.grav_mode || a.wb || a.tc)
    return launch_step_recon<T, RS, FORM_SOURCES>(recon, grid, s, t0, t1, a);
  return launch_step_recon<T, RS, FORM_PLAIN>(recon, grid, s, t0, t1, a);
}

template <int RS>
cudaError_t launch_step_rs(int tile, int recon, dim3 grid, cudaStream_t s, const CUtensorMap &t0,
                           const CUtensorMap &t1, const StepArgs &a) {
  return tile == TILE_SMALL ? launch_step_form<SmallTile, RS>(recon, grid, s, t0, t1, a)
                            : launch_step_form<WideTile, RS>(recon, grid, s, t0, t1, a);
}

}  // namespace fv2d
