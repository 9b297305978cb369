// The pixel pass of an iteration with the odd compile-time plans, FP32, finite strain.
#include "disp_launch.cuh"

namespace musg {

bool disp_odd_pixels_finite(int tk, const TilePlan &pl, const DispArgs<float> &a, const DispShape &c, int B, cudaStream_t s) {
  switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, BB)                                                                          \
  case M:                                                                                         \
    if (tk == TK_FISO)                                                                            \
      disp_launch<float>(k_pixels<float, 3, true, TK_FISO, IN_SPEC, OUT_SPEC, A, BB, false>, a, c, B, s); \
    else                                                                                          \
      disp_launch<float>(k_pixels<float, 3, true, TK_ANYFIN, IN_SPEC, OUT_SPEC, A, BB, false>, a, c, B, s); \
    return true;
    MUSG_DISP_PLANS_ODD(MUSG_C)
#undef MUSG_C
    default: return false;
  }
}

}  // namespace musg
