// The order of the service's copies between its streams, with the runtime of
// fake_cudart.hpp: starts a server with the autotuner's trials, submits requests
// in bursts, and stops it.  Prints the races found; exit code 0: none.
#include <chrono>
#include <thread>

#include "../include/fv2d_gpu.h"
#include "../include/fv2d_serve.h"
#include "fake_cudart.hpp"

int main() {
  fv2d_server_config cfg = {};
  cfg.struct_size = sizeof cfg;
  cfg.budget_bytes = 2e9;
  cfg.max_sims = 64;
  cfg.autotune = 1;
  fv2d_server *s = nullptr;
  if (fv2d_server_create(&cfg, &s) != FV2D_OK) return 2;
  {
    std::lock_guard<std::mutex> lock(fake::rt().mu);
    if (fake::rt().copies.empty() || fake::rt().launches.empty()) return 3;  // no trial ran
  }
  for (int burst = 0; burst < 3; ++burst) {
    fv2d_server_stats before, st;
    fv2d_server_get_stats(s, &before);
    for (int k = 0; k < 6; ++k) {
      fv2d_request r = {};
      r.struct_size = sizeof r;
      r.problem = FV2D_PB_KH_STEP;
      fv2d_params_default(&r.params);
      r.params.Nx = 32 + 16 * k;
      r.params.Ny = 24;
      r.max_steps = 100;
      int64_t id;
      if (fv2d_server_submit(s, &r, &id) != FV2D_OK) return 4;
    }
    for (int wait = 0; wait < 20000; ++wait) {  // all admitted, and a few replays on
      fv2d_server_get_stats(s, &st);
      if (st.admitted == 6 * (burst + 1) && st.replays >= before.replays + 3) break;
      std::this_thread::sleep_for(std::chrono::milliseconds(1));
    }
    if (st.admitted != 6 * (burst + 1)) return 5;
  }
  fv2d_server_destroy(s);
  for (const std::string &r : fake::rt().races) std::printf("%s\n", r.c_str());
  return fake::rt().races.empty() ? 0 : 1;
}
