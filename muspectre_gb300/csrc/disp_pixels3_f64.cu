// The displacement-space CG's pixel pass in 3-D, FP64.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS(double, 3)
MUSG_INSTANTIATE_PIXELS_IO(double, 3)
}  // namespace musg
