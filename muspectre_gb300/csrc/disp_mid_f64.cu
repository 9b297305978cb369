// The passes of disp_mid.cuh in FP64.
#include "disp_mid.cuh"

namespace musg {
MUSG_INSTANTIATE_DISP_MID(double)
}  // namespace musg
