// The displacement-space CG's pixel pass in 2-D, FP64.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS(double, 2)
}  // namespace musg
