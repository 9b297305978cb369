// Out-of-line tile transforms, FP32, 3-D grids.
#include "tile_stages.cuh"

namespace musg {

__device__ __noinline__ bool tile_fft_rt(bool inv, int n, int m, int r1, int r2, int nst, unsigned long long rcode, int blu,
                                         const float2 *tw, const float2 *chirp, const float2 *bf, const TileLay lay, uint32_t buf,
                                         uint32_t buf2, int P, uint32_t tws) {
  return tile_fft_any<float2, false>(inv, n, m, r1, r2, nst, rcode, blu, tw, chirp, bf, lay, buf, buf2, P, tws);
}

}  // namespace musg
