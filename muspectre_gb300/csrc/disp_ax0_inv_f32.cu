// The passes of disp_ax0_inv.cuh in FP32.
#include "disp_ax0_inv.cuh"

namespace musg {
MUSG_INSTANTIATE_DISP_AX0_INV(float)
}  // namespace musg
