// The pixel pass in 2-D from and to real fields, FP32.
#include "disp_pixels.cuh"

namespace musg {
MUSG_INSTANTIATE_PIXELS_IO(float, 2)
}  // namespace musg
