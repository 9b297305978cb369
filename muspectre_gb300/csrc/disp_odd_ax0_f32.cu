// The axis-0 passes of an iteration with the odd compile-time plans, FP32.
#include "disp_launch.cuh"

namespace musg {

bool disp_odd_ax0(bool fin, bool step, const TilePlan &pl, const DispArgs<float> &a, const DispShape &c, int B, cudaStream_t s) {
  switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, BB)                                                                          \
  case M:                                                                                         \
    if (fin) {                                                                                    \
      if (step)                                                                                   \
        disp_launch<float>(k_ax0_inv<float, 3, true, AX_STEP, A, BB, false>, a, c, B, s);         \
      else                                                                                        \
        disp_launch<float>(k_ax0_fwd<float, 3, true, AX_DOTS, A, BB, false>, a, c, B, s);         \
    } else {                                                                                      \
      if (step)                                                                                   \
        disp_launch<float>(k_ax0_inv<float, 3, false, AX_STEP, A, BB, false>, a, c, B, s);        \
      else                                                                                        \
        disp_launch<float>(k_ax0_fwd<float, 3, false, AX_DOTS, A, BB, false>, a, c, B, s);        \
    }                                                                                             \
    return true;
    MUSG_DISP_PLANS_ODD(MUSG_C)
#undef MUSG_C
    default: return false;
  }
}

}  // namespace musg
