// The axis-1 passes of an iteration with the odd compile-time plans, FP32.
#include "disp_launch.cuh"

namespace musg {

bool disp_odd_mid(bool fin, bool inv, const TilePlan &pl, const DispArgs<float> &a, const DispShape &c, int B, cudaStream_t s) {
  switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, BB)                                                                          \
  case M:                                                                                         \
    if (fin) {                                                                                    \
      if (inv)                                                                                    \
        disp_launch<float>(k_mid<float, true, true, A, BB, false>, a, c, B, s);                   \
      else                                                                                        \
        disp_launch<float>(k_mid<float, true, false, A, BB, false>, a, c, B, s);                  \
    } else {                                                                                      \
      if (inv)                                                                                    \
        disp_launch<float>(k_mid<float, false, true, A, BB, false>, a, c, B, s);                  \
      else                                                                                        \
        disp_launch<float>(k_mid<float, false, false, A, BB, false>, a, c, B, s);                 \
    }                                                                                             \
    return true;
    MUSG_DISP_PLANS_ODD(MUSG_C)
#undef MUSG_C
    default: return false;
  }
}

}  // namespace musg
