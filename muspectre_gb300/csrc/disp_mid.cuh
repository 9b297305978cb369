// Launches of the displacement-space CG's axis-1 passes (disp.cuh).
#pragma once

#include "disp_launch.cuh"

namespace musg {
namespace {

template <typename R, bool FIN, bool INV>
void mid(const TilePlan &pl, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s, const DispGroup<R> *grp) {
  if (grp) return disp_launch<R>(k_mid<R, FIN, INV, (kGroupPlan<R, 3>), (kGroupPlan<R, 3>), true>, a, c, B, s, grp);
  if constexpr (sizeof(R) == 4) {
    switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, BB) \
  case M: return disp_launch<R>(k_mid<R, FIN, INV, A, BB, false>, a, c, B, s);
      MUSG_DISP_PLANS(MUSG_C)
#undef MUSG_C
      default:
        if (disp_odd_mid(FIN, INV, pl, a, c, B, s)) return;
    }
  }
  disp_launch<R>(k_mid<R, FIN, INV, 0, 0, false>, a, c, B, s);
}
}  // namespace

template <typename R>
void disp_mid(const Spectral &sp, bool inv, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
             const DispGroup<R> *grp) {
  const TilePlan &pl = sp.tile<R>(1);
  if (disp_finite(sp)) inv ? mid<R, true, true>(pl, a, c, B, s, grp) : mid<R, true, false>(pl, a, c, B, s, grp);
  else inv ? mid<R, false, true>(pl, a, c, B, s, grp) : mid<R, false, false>(pl, a, c, B, s, grp);
}

#define MUSG_INSTANTIATE_DISP_MID(R) \
template void disp_mid<R>(const Spectral &, bool, const DispArgs<R> &, const DispShape &, int, cudaStream_t, \
                              const DispGroup<R> *);

}  // namespace musg
