// The displacement-space CG's pixel pass in 3-D, FP32.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS(float, 3)
MUSG_INSTANTIATE_PIXELS_IO(float, 3)
}  // namespace musg
