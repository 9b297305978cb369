// Host check of the FFT plans of the displacement-space passes: every axis length whose
// shortest 7-smooth plan fits the shared memory of a block gets a plan that fits its
// passes too, and radices above 17 appear only where no two up to 17 make the length.
// Prints the lengths that fail; exit status 1 if there are any.
#include <algorithm>
#include <cstdio>

#include "musg_internal.h"

using namespace musg;

static bool smooth(int v) {
  for (int p : {2, 3, 5, 7})
    while (v % p == 0) v /= p;
  return v == 1;
}

int main() {
  const long bytes = 232448 - 2048;  // 227 KB less the static arrays
  int bad = 0, checked = 0, longest[2][2][3] = {};
  for (int dim = 2; dim <= 3; ++dim)
    for (int small = 0; small < 2; ++small)
      for (int axis = 0; axis < dim; ++axis) {
        const int sym = dim * (dim + 1) / 2, all = dim * dim;
        const bool middle = dim == 3 && axis == 1;
        const int pencils = middle ? 1 : axis == 0 ? (small ? sym : 2) : small ? sym : all;
        for (int n = 1; n <= 7300; ++n) {
          int ms = n;
          if (!smooth(n))
            for (ms = 2 * n - 1; !smooth(ms);) ++ms;
          if ((middle ? 1L : all) * ms * 32 > bytes) continue;  // all components of a pencil, two buffers
          Spectral sp;
          sp.g.dim = dim;
          sp.proj_kind = small ? MUSG_PROJ_SMALL_STRAIN : MUSG_PROJ_FINITE_STRAIN;
          TilePlan t;
          t.factor(n, dim == 2 ? 32 : 17, wide_bluestein<double>(n, dim), sp.tile_points<double>(axis, bytes));
          // two stages: one buffer, its groups of r1 slots padded by at most 15 each way
          const long row = t.r1 ? (long)t.r2 * (t.r1 + 15) + 15 : 2L * t.m;
          const long need = 16 * (pencils * row + (t.r1 ? t.m : 0));
          ++checked;
          longest[dim - 2][small][axis] = std::max(longest[dim - 2][small][axis], n);
          if (!t.m || need > bytes || (t.blu && t.m < 2 * n - 1)) {
            std::printf("dim %d small %d axis %d: length %d, plan %d (%d factors), %ld bytes\n", dim, small, axis, n, t.m,
                        t.nst, need);
            ++bad;
          }
        }
      }
  for (int n = 1; n <= 1024; ++n) {
    TilePlan t;
    t.factor(n, 32, 32, 1 << 28);
    bool narrow = false;
    for (int a = 1; a <= 17; ++a) narrow |= n % a == 0 && n / a <= 17;
    if (narrow && (t.blu || t.nst != 2 || t.r1 > 17)) {
      std::printf("length %d: %d x %d\n", n, t.r1, t.r2);
      ++bad;
    }
  }
  std::printf("%d lengths checked, %d refused\n", checked, bad);
  return bad ? 1 : 0;
}
