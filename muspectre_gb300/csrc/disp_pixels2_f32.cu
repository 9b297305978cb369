// The displacement-space CG's pixel pass in 2-D, FP32.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS(float, 2)
}  // namespace musg
