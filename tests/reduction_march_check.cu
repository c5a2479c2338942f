// Host check of the planes that the diagnostics' reduction asks L2 for
// (red_ahead_plane): for every grid depth and march length, every plane asked for
// lies in the grid and is one that the march loads later, and every plane that a
// step after the first RED_AHEAD of a march loads as the cell above it has been
// asked for.  Built and run by tests/test_reduction_march.py.
#include <cstdio>

#include "aux_kernels.cuh"

using namespace wdm;

int main() {
  int failures = 0;
  for (int nz : {8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512})
    for (int depth : {4, 8, 16, 32})
      for (int z0 = 0; z0 < nz; z0 += depth) {
        const int z1 = z0 + depth < nz ? z0 + depth : nz;
        for (int z = z0; z < z1; ++z) {
          const int p = red_ahead_plane(z, z1, nz);
          const int step = z + RED_AHEAD;  // the step that loads it, plane step + 1
          const bool loads = step < z1 && step + 1 < nz;
          if (p >= nz || p != (loads ? step + 1 : -1)) {
            std::printf("nz=%d march %d..%d step %d: plane %d\n", nz, z0, z1, z, p);
            ++failures;
          }
        }
      }
  std::printf("%s\n", failures ? "FAILED" : "ALL OK");
  return failures ? 1 : 0;
}
