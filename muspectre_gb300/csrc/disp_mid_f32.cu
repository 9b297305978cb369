// The passes of disp_mid.cuh in FP32.
#include "disp_mid.cuh"

namespace musg {
MUSG_INSTANTIATE_DISP_MID(float)
}  // namespace musg
