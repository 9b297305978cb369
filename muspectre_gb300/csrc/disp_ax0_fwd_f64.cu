// The passes of disp_ax0_fwd.cuh in FP64.
#include "disp_ax0_fwd.cuh"

namespace musg {
MUSG_INSTANTIATE_DISP_AX0_FWD(double)
}  // namespace musg
