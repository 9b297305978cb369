// The pixel pass in 2-D from and to real fields, FP64.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS_IO(double, 2)
}  // namespace musg
