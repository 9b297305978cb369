// Out-of-line tile transforms (tile_fft.cuh): every role of every radix, compiled once
// and called by the kernels of the displacement-space CG through tile_fft_rt (relocatable
// device code): all roles inline in every kernel were ten minutes of compilation.
// Included by tile_stages_f32.cu and tile_stages_f64.cu (3-D) and their tile_stages2_ twins (2-D).
#pragma once

#include "tile_fft.cuh"

namespace musg {
namespace {

template <typename T, int RAD, int OP>
__device__ __noinline__ void tile_stage_rt(uint32_t buf, uint32_t tw, const TileLay lay, const TileStageArgs<T> a) {
  const WinBuf<T> b{buf};
  tile_stage<RAD, OP, T>(lay, WinBuf<T>{tw}, a, [&](int, int s, int p) { return b.ld(lay.at(s, p)); },
                         [&](int, int s, int p, T v) { b.st(lay.at(s, p), v); });
}

template <typename T, int OP, bool WIDE>
__device__ __forceinline__ void tile_stage_any(int rad, uint32_t buf, uint32_t tw, const TileLay &lay,
                                               const TileStageArgs<T> &a) {
  switch (rad) {
#define MUSG_TS(RAD) \
  case RAD: tile_stage_rt<T, RAD, OP>(buf, tw, lay, a); break;
    MUSG_TILE_RADICES(MUSG_TS)
#undef MUSG_TS
#define MUSG_TS(RAD) \
  case RAD: if constexpr (WIDE) tile_stage_rt<T, RAD, OP>(buf, tw, lay, a); break;
    MUSG_TILE_RADICES_2D(MUSG_TS)
#undef MUSG_TS
    default: tile_stage_rt<T, 1, OP>(buf, tw, lay, a); break;
  }
}

// one out-of-place Stockham stage (natural order) of a plan of three or more factors:
// the formulation of fft_device.cuh
template <typename T, int RAD, bool INV>
__device__ __noinline__ void tile_stockham_rt(uint32_t src_, uint32_t dst_, const T *__restrict__ tw, const TileLay lay,
                                              int P, int m, int Ns) {
  const WinBuf<T> src{src_}, dst{dst_};
  const int nb = m / RAD, tws = m / (Ns * RAD);
  const FDiv fNs(Ns);
  lay.each(nb, P, [&](int j, int p) {
    int k;
    fNs.div(j, k);
    T v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) v[r] = src.ld(lay.at(j + r * nb, p));
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) v[r] = cmul(v[r], conj_if(__ldg(&tw[k * r * tws]), INV));
    }
    Dft<RAD, INV, T>::run(v);
    const int o = (j - k) * RAD + k;
#pragma unroll
    for (int r = 0; r < RAD; ++r) dst.st(lay.at(o + r * Ns, p), v[r]);
  });
}

template <typename T, bool INV>
__device__ __forceinline__ bool tile_multi(int m, int nst, unsigned long long code, const T *tw, const TileLay lay,
                                           uint32_t src, uint32_t dst, int P) {
  int Ns = 1;
  for (int s = 0; s < nst; ++s, code >>= 5) {
    const int rad = (int)(code & 31ull);
    switch (rad) {
#define MUSG_SH(RAD) \
  case RAD: tile_stockham_rt<T, RAD, INV>(src, dst, tw, lay, P, m, Ns); break;
      MUSG_SH(2) MUSG_SH(3) MUSG_SH(4) MUSG_SH(5) MUSG_SH(6) MUSG_SH(7) MUSG_SH(8) MUSG_SH(9) MUSG_SH(10)
      MUSG_SH(11) MUSG_SH(12) MUSG_SH(13) MUSG_SH(14) MUSG_SH(15) MUSG_SH(16)
#undef MUSG_SH
      default: tile_stockham_rt<T, 17, INV>(src, dst, tw, lay, P, m, Ns); break;
    }
    __syncthreads();
    Ns *= rad;
    const uint32_t t = src;
    src = dst;
    dst = t;
  }
  return (nst & 1) != 0;
}

template <typename T, bool WIDE>
__device__ __forceinline__ bool tile_fft_any(bool inv, int n, int m, int r1, int r2, int nst, unsigned long long rcode,
                                             int blu, const T *tw, const T *chirp, const T *bf, const TileLay lay,
                                             uint32_t buf, uint32_t buf2, int P, uint32_t tws) {
  if (r1) {
    TileStageArgs<T> a{P, r2, lay.S, n, inv ? 1 : 0, chirp, bf};  // radix r1
    TileStageArgs<T> c = a;                                     // radix r2
    c.ra = r1;
    if (blu) {
      tile_stage_any<T, OP_B1, WIDE>(r1, buf, tws, lay, a);
      __syncthreads();
      tile_stage_any<T, OP_BM, WIDE>(r2, buf, tws, lay, c);
      __syncthreads();
      tile_stage_any<T, OP_B2, WIDE>(r1, buf, tws, lay, a);
    } else if constexpr (!WIDE) {  // (2-D kernels have these stages inline)
      if (inv) {
        tile_stage_any<T, OP_I1, WIDE>(r2, buf, tws, lay, c);
        __syncthreads();
        tile_stage_any<T, OP_I2, WIDE>(r1, buf, tws, lay, a);
      } else {
        tile_stage_any<T, OP_F1, WIDE>(r1, buf, tws, lay, a);
        __syncthreads();
        tile_stage_any<T, OP_F2, WIDE>(r2, buf, tws, lay, c);
      }
    }
    __syncthreads();
    return false;
  }
  if (!blu)
    return inv ? tile_multi<T, true>(m, nst, rcode, tw, lay, buf, buf2, P)
               : tile_multi<T, false>(m, nst, rcode, tw, lay, buf, buf2, P);
  // Bluestein over three or more factors, natural order
  auto each = [&](auto f) {
    lay.each(m, P, [&](int e, int p) { f(e, lay.at(e, p)); });
    __syncthreads();
  };
  const WinBuf<T> x{buf};
  each([&](int e, int o) { x.st(o, e < n ? cmul(conj_if(x.ld(o), inv), __ldg(&chirp[e])) : T{0, 0}); });
  const bool second = tile_multi<T, false>(m, nst, rcode, tw, lay, buf, buf2, P);
  const uint32_t cb = second ? buf2 : buf, db = second ? buf : buf2;
  const WinBuf<T> c{cb};
  each([&](int e, int o) { c.st(o, cmul(c.ld(o), __ldg(&bf[e]))); });
  const bool swapped = tile_multi<T, true>(m, nst, rcode, tw, lay, cb, db, P);
  const WinBuf<T> d{swapped ? db : cb};
  each([&](int e, int o) {
    if (e < n) d.st(o, conj_if(cmul(d.ld(o), __ldg(&chirp[e])), inv));
  });
  return swapped != second;
}

}  // namespace

}  // namespace musg
