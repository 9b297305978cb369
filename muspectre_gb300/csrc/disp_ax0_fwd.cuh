// Launches of the displacement-space CG's axis-0 forward passes (disp.cuh): with the
// iteration's sums, and the plain contraction.
#pragma once

#include "disp_launch.cuh"

namespace musg {
namespace {

template <typename R, int D, bool FIN>
void ax0_dots(const TilePlan &pl, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
              const DispGroup<R> *grp) {
  if (grp) return disp_launch<R>(k_ax0_fwd<R, D, FIN, AX_DOTS, (kGroupPlan<R, D>), (kGroupPlan<R, D>), true>, a, c, B, s, grp);
  if constexpr (sizeof(R) == 4) {
    switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, BB) \
  case M: return disp_launch<R>(k_ax0_fwd<R, D, FIN, AX_DOTS, A, BB, false>, a, c, B, s);
      MUSG_DISP_PLANS(MUSG_C)
#undef MUSG_C
      default:
        if constexpr (D == 3)
          if (disp_odd_ax0(FIN, false, pl, a, c, B, s)) return;
    }
  }
  disp_launch<R>(k_ax0_fwd<R, D, FIN, AX_DOTS, kRtPlan<D>, kRtPlan<D>, false>, a, c, B, s);
}
}  // namespace

template <typename R>
void disp_ax0_dots(const Spectral &sp, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
              const DispGroup<R> *grp) {
  const bool fin = disp_finite(sp);
  if (sp.g.dim == 2) fin ? ax0_dots<R, 2, true>(sp.tile<R>(0), a, c, B, s, grp) : ax0_dots<R, 2, false>(sp.tile<R>(0), a, c, B, s, grp);
  else fin ? ax0_dots<R, 3, true>(sp.tile<R>(0), a, c, B, s, grp) : ax0_dots<R, 3, false>(sp.tile<R>(0), a, c, B, s, grp);
}

template <typename R>
void disp_ax0_contract(const Spectral &sp, const DispArgs<R> &a, const DispShape &c, cudaStream_t s) {
#define MUSG_C(DD, FF) \
  if (sp.g.dim == DD && disp_finite(sp) == FF) disp_launch<R>(k_ax0_fwd<R, DD, FF, AX_OUT, kRtPlan<DD>, kRtPlan<DD>, false>, a, c, 1, s);
  MUSG_C(2, true) MUSG_C(2, false) MUSG_C(3, true) MUSG_C(3, false)
#undef MUSG_C
}

#define MUSG_INSTANTIATE_DISP_AX0_FWD(R) \
template void disp_ax0_dots<R>(const Spectral &, const DispArgs<R> &, const DispShape &, int, cudaStream_t, \
                                   const DispGroup<R> *); \
template void disp_ax0_contract<R>(const Spectral &, const DispArgs<R> &, const DispShape &, cudaStream_t);

}  // namespace musg
