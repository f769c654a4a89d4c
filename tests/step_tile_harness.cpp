// The FP64 step's tile and its overlapped launches on devices of different SM
// counts, with the runtime of fake_cudart.hpp.  Reads lines "SMs Nx Ny", prints for
// each the tile's side (8 or 16) and whether a device loop's launches overlap.
#include "../include/fv2d_gpu.h"
#include "fake_cudart.hpp"

int main() {
  int sms, nx, ny;
  while (std::scanf("%d %d %d", &sms, &nx, &ny) == 3) {
    fake::Runtime &r = fake::rt();
    r.sms = sms;
    fv2d_params p;
    fv2d_params_default(&p);
    p.Nx = nx;
    p.Ny = ny;
    fv2d_ctx *c = nullptr;
    if (fv2d_create(&p, 0, &c) != FV2D_OK || fv2d_init_problem(c, FV2D_PB_SOD_X) != FV2D_OK) return 2;
    r.launches.clear();
    if (fv2d_run_async(c, 1) != FV2D_OK) return 3;
    int side = 0, overlap = 0;
    for (const fake::Launch &l : r.launches)
      if (l.kernel.find("step_kernel") != std::string::npos) {
        side = l.kernel.find("ILi8ELi8E") != std::string::npos ? 8 : 16;
        overlap = l.programmatic;
      }
    std::printf("%d %d\n", side, overlap);
    fv2d_destroy(c);
  }
  return 0;
}
