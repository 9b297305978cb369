// Launches of the displacement-space CG's pixel pass (disp.cuh) for one dimension,
// included by the disp_pixels*.cu (the iteration's
// pass and the ones from and to real fields build side by side where they are long to build).
#pragma once

#include "disp_launch.cuh"

namespace musg {
namespace {

template <typename R, int D, bool FIN, int TK>
void pixels_iteration(const TilePlan &pl, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
                      const DispGroup<R> *grp) {
  if (grp) {
    disp_launch<R>(k_pixels<R, D, FIN, TK, IN_SPEC, OUT_SPEC, (kGroupPlan<R, D>), (kGroupPlan<R, D>), true>, a, c, B, s, grp);
    return;
  }
  if constexpr (sizeof(R) == 4) {
    switch (disp_fixed_plan(pl)) {
#define MUSG_PX(M, A, BB) \
  case M: disp_launch<R>(k_pixels<R, D, FIN, TK, IN_SPEC, OUT_SPEC, A, BB, false>, a, c, B, s); return;
      MUSG_DISP_PLANS(MUSG_PX)
#undef MUSG_PX
      default:
        if constexpr (D == 3 && FIN)
          if (disp_odd_pixels_finite(TK, pl, a, c, B, s)) return;
        if constexpr (D == 3 && !FIN)
          if (disp_odd_pixels_small(TK, pl, a, c, B, s)) return;
    }
  }
  disp_launch<R>(k_pixels<R, D, FIN, TK, IN_SPEC, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, B, s);
}

}  // namespace

// kernels of their own for the isotropic laws (LE1, LE3, LE4; FP64 stores S, FP32 rebuilds
// it) and the generic small-strain stiffness; the other finite-strain kinds share one
// that picks per launch
template <typename R, int D>
void disp_pixels(int tkind, const TilePlan &pl, const DispArgs<R> &a0, const DispShape &c, int B, cudaStream_t s,
                 const DispGroup<R> *grp) {
  DispArgs<R> a = a0;
  a.tkind = tkind;
  switch (tkind) {
    case TK_SMALL: return pixels_iteration<R, D, false, TK_SMALL>(pl, a, c, B, s, grp);
    case TK_GSMALL: return pixels_iteration<R, D, false, TK_GSMALL>(pl, a, c, B, s, grp);
    case sizeof(R) == 4 ? TK_FISO : TK_FINITE:
      return pixels_iteration<R, D, true, sizeof(R) == 4 ? TK_FISO : TK_FINITE>(pl, a, c, B, s, grp);
    default: return pixels_iteration<R, D, true, TK_ANYFIN>(pl, a, c, B, s, grp);
  }
}

template <typename R, int D>
void disp_pixels_in(bool fin, int tkind, bool delta, const DispArgs<R> &a0, const DispShape &c, cudaStream_t s) {
  DispArgs<R> a = a0;
  a.tkind = tkind;
  if (tkind == TK_PLAIN) {
    if (fin && delta) disp_launch<R>(k_pixels<R, D, true, TK_PLAIN, IN_DELTA, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
    else if (fin) disp_launch<R>(k_pixels<R, D, true, TK_PLAIN, IN_REAL, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
    else if (delta) disp_launch<R>(k_pixels<R, D, false, TK_PLAIN, IN_DELTA, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
    else disp_launch<R>(k_pixels<R, D, false, TK_PLAIN, IN_REAL, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
  } else if (tkind == TK_SMALL) {
    disp_launch<R>(k_pixels<R, D, false, TK_SMALL, IN_REAL, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
  } else if (tkind == TK_GSMALL) {
    disp_launch<R>(k_pixels<R, D, false, TK_GSMALL, IN_REAL, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
  } else {
    disp_launch<R>(k_pixels<R, D, true, TK_ANYFIN, IN_REAL, OUT_SPEC, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
  }
}

template <typename R, int D>
void disp_pixels_out(bool fin, const DispArgs<R> &a, const DispShape &c, cudaStream_t s) {
  if (fin) disp_launch<R>(k_pixels<R, D, true, TK_PLAIN, IN_SPEC, OUT_REAL, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
  else disp_launch<R>(k_pixels<R, D, false, TK_PLAIN, IN_SPEC, OUT_REAL, kRtPlan<D>, kRtPlan<D>, false>, a, c, 1, s);
}

#define MUSG_INSTANTIATE_PIXELS(R, D)                                                                             \
  template void disp_pixels<R, D>(int, const TilePlan &, const DispArgs<R> &, const DispShape &, int, cudaStream_t, \
                                  const DispGroup<R> *);
#define MUSG_INSTANTIATE_PIXELS_IO(R, D)                                                                          \
  template void disp_pixels_in<R, D>(bool, int, bool, const DispArgs<R> &, const DispShape &, cudaStream_t);      \
  template void disp_pixels_out<R, D>(bool, const DispArgs<R> &, const DispShape &, cudaStream_t);

}  // namespace musg
