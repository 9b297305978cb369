// The passes of disp_ax0_fwd.cuh in FP32.
#include "disp_ax0_fwd.cuh"

namespace musg {
MUSG_INSTANTIATE_DISP_AX0_FWD(float)
}  // namespace musg
