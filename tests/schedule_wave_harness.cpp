// Runs choose_wave_band (fv2d_gb300/csrc/schedule.hpp) on cases read from
// stdin: a line "n warps" then n lines "strips Ny" each; prints the band height
// of each case.
#include <cstdio>
#include <vector>

#include "../fv2d_gb300/csrc/schedule.hpp"

int main() {
  int n;
  double warps;
  while (std::scanf("%d %lf", &n, &warps) == 2) {
    std::vector<fv2d::BandGrid> g(n);
    for (auto &x : g)
      if (std::scanf("%d %d", &x.strips, &x.Ny) != 2) return 2;
    std::printf("%d\n", fv2d::choose_wave_band(g, warps));
  }
  return 0;
}
