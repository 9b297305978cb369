// Register-resident pencil FFT passes for power-of-two lengths 16..256 (device code).
//
// A length M = R1 * R2 (R2 divides R1) transform is the two-stage Stockham network of
// fft_device.cuh with a fixed thread mapping instead of a loop over butterflies:
//   stage 1: lane y < Y = M / R1 holds x[y + Y r] (r < R1) in registers straight from
//            global memory, applies DFT_R1 and writes slot y R1 + r of its pencil in
//            shared memory;
//   stage 2: after one barrier, lane y takes the butterflies j = y + Y b (b < R1 / R2):
//            inputs slot j + R1 r (r < R2), twiddles W_M^(j r), DFT_R2, giving X[j + R1 r],
//            stored straight to global memory (or kept for the Green operator).
// The unnormalised inverse is the adjoint network in mirror order: IDFT_R2 of
// X[j + R1 r] followed by the conjugate twiddles, written back to the same slots; one
// barrier; IDFT_R1 of slots y R1 + r gives x[y + Y r].  Every index is a compile-time
// constant or a multiply-add of the thread coordinates, the radices are unrolled, and
// shared memory holds one buffer (no ping-pong), so a block keeps more pencils in
// flight than the generic path.
//
// Thread block: (T pencils of a tile, Y lanes, NC components); the pencils of a tile are
// T consecutive positions of the contiguous inner extent, so a warp reads and writes
// rows of T consecutive complex values.
#pragma once

#include "spectral.cuh"

namespace musg {

template <int M> struct RegPlan;
template <> struct RegPlan<16> { static constexpr int R1 = 4, R2 = 4; };
template <> struct RegPlan<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct RegPlan<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct RegPlan<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct RegPlan<256> { static constexpr int R1 = 16, R2 = 16; };

template <int M> struct RegFft {
  static constexpr int R1 = RegPlan<M>::R1, R2 = RegPlan<M>::R2;
  static constexpr int Y = M / R1;
  static constexpr int NB = R1 / R2;
  static_assert(R1 * R2 == M && R1 % R2 == 0 && Y == R2, "two-stage plan");
};

inline bool reg_fft_length(int m) { return m == 16 || m == 32 || m == 64 || m == 128 || m == 256; }

// stage-2 twiddle W_M^(j r) (j < R1, r < R2, so j r < M) from the block's shared
// copy of the plan's table (stage_twiddles)
template <bool CONJ, typename T>
__device__ __forceinline__ T reg_tw(const T *tw, int idx) {
  T w = tw[idx];
  if (CONJ) w.y = -w.y;
  return w;
}

// copy the plan's twiddle table W_M^k (k < M) into shared memory, by the whole block;
// a barrier must separate it from the first reg_tw.  Per-thread loads of the table
// from global memory (L1 hits) made the stage-2 butterflies wait on the load pipe:
// the last-axis inverse ran 63.5 us with them and 49.2 us with the shared copy.
template <int M, typename T>
__device__ __forceinline__ void stage_twiddles(T *dst, const T *__restrict__ src) {
  for (int k = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z); k < M;
       k += blockDim.x * blockDim.y * blockDim.z)
    dst[k] = src[k];
}

// ------------------------------------------------------------ middle-axis pass
// pencils along axis 1 of [c][k0][k1][k2h]: AxisArgs as for k_axis, blockIdx.x =
// tile + ntiles * slab, blockIdx.z = problem of a batched launch
template <typename R, int M, bool INV>
__global__ void __launch_bounds__(512) k_axis_reg(const AxisArgs<R> a0) {
  dep_wait();
  using T = typename V2<R>::T;
  using F = RegFft<M>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *buf = reinterpret_cast<T *>(smem_raw);
  AxisArgs<R> a = a0;
  if (a0.batch) {
    a.spec = a0.batch[blockIdx.z].spec;
    a.st = a0.batch[blockIdx.z].st;
  }
  if (a.st && !a.st->active) return;
  const int Tt = blockDim.x, t = threadIdx.x, y = threadIdx.y;
  T *tws = buf + (size_t)Tt * M;  // after the tile
  stage_twiddles<M>(tws, a.ap.tw);
  const int tile = blockIdx.x % a.ntiles;
  const long long slab = blockIdx.x / a.ntiles;
  const long long pos = (long long)tile * Tt + t;
  const bool ok = pos < a.inner;
  T *base = a.spec + slab * a.sb + pos;
  const long long se = a.se;
  if (!INV) {
    T v[F::R1];
#pragma unroll
    for (int r = 0; r < F::R1; ++r) v[r] = ok ? base[(y + F::Y * r) * se] : T{R(0), R(0)};
    Dft<F::R1, false, T>::run(v);
#pragma unroll
    for (int r = 0; r < F::R1; ++r) buf[(y * F::R1 + r) * Tt + t] = v[r];
    __syncthreads();
#pragma unroll
    for (int b = 0; b < F::NB; ++b) {
      const int j = y + F::Y * b;
      T w[F::R2];
#pragma unroll
      for (int r = 0; r < F::R2; ++r) w[r] = buf[(j + F::R1 * r) * Tt + t];
#pragma unroll
      for (int r = 1; r < F::R2; ++r) w[r] = cmul(w[r], reg_tw<false>(tws, j * r));
      Dft<F::R2, false, T>::run(w);
      if (ok) {
#pragma unroll
        for (int r = 0; r < F::R2; ++r) base[(j + F::R1 * r) * se] = w[r];
      }
    }
  } else {
    __syncthreads();  // the twiddle copy
#pragma unroll
    for (int b = 0; b < F::NB; ++b) {
      const int j = y + F::Y * b;
      T w[F::R2];
#pragma unroll
      for (int r = 0; r < F::R2; ++r) w[r] = ok ? base[(j + F::R1 * r) * se] : T{R(0), R(0)};
      Dft<F::R2, true, T>::run(w);
#pragma unroll
      for (int r = 1; r < F::R2; ++r) w[r] = cmul(w[r], reg_tw<true>(tws, j * r));
#pragma unroll
      for (int r = 0; r < F::R2; ++r) buf[(j + F::R1 * r) * Tt + t] = w[r];
    }
    __syncthreads();
    T v[F::R1];
#pragma unroll
    for (int r = 0; r < F::R1; ++r) v[r] = buf[(y * F::R1 + r) * Tt + t];
    Dft<F::R1, true, T>::run(v);
    if (ok) {
#pragma unroll
      for (int r = 0; r < F::R1; ++r) base[(y + F::Y * r) * se] = v[r];
    }
  }
}

// ------------------------------------------------------------ Green pass
// first-axis forward FFT, Green operator, first-axis inverse FFT on the spectrum
// [c][k0][rho] (rho = k1 * nh + k2 in 3-D, k1 in 2-D).  Finite strain couples the D
// components of one row i of the tensor only: blockIdx.y = i, threadIdx.z = j picks
// component i + D j.  Small strain couples all D^2: threadIdx.z = component,
// gridDim.y = 1.  blockIdx.z = problem of a batched launch.  Shared memory:
// slot-major [slot][z][t], NC * T pencils of M entries.
template <typename R, int M, int MODE, int D>
__global__ void __launch_bounds__(384, 2) k_green_reg(const GreenArgs<R> a0) {
  dep_wait();
  using T = typename V2<R>::T;
  using F = RegFft<M>;
  static_assert(MODE == GM_SMALL || MODE == GM_FINITE, "projection modes only");
  constexpr int NC = MODE == GM_FINITE ? D : D * D;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *buf = reinterpret_cast<T *>(smem_raw);
  GreenArgs<R> a = a0;
  if (a0.batch) {
    a.spec = a0.batch[blockIdx.z].spec;
    a.st = a0.batch[blockIdx.z].st;
  }
  if (a.st && !a.st->active) return;
  const int Tt = blockDim.x, t = threadIdx.x, y = threadIdx.y, z = threadIdx.z;
  const int P = NC * Tt;
  const int comp = MODE == GM_FINITE ? (int)blockIdx.y + D * z : z;
  const long long rho = (long long)blockIdx.x * Tt + t;
  const bool ok = rho < a.Rr;
  T *base = a.spec + (long long)comp * a.nk + rho;
  const long long se = a.Rr;
  T *col = buf + z * Tt + t;  // this thread's pencil: slot s at col[s * P]
  T *tws = buf + (size_t)P * M;  // after the tile
  stage_twiddles<M>(tws, a.ap.tw);
  {
    T v[F::R1];
#pragma unroll
    for (int r = 0; r < F::R1; ++r) v[r] = ok ? base[(y + F::Y * r) * se] : T{R(0), R(0)};
    Dft<F::R1, false, T>::run(v);
#pragma unroll
    for (int r = 0; r < F::R1; ++r) col[(y * F::R1 + r) * P] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < F::NB; ++b) {
    const int j = y + F::Y * b;
    T w[F::R2];
#pragma unroll
    for (int r = 0; r < F::R2; ++r) w[r] = col[(j + F::R1 * r) * P];
#pragma unroll
    for (int r = 1; r < F::R2; ++r) w[r] = cmul(w[r], reg_tw<false>(tws, j * r));
    Dft<F::R2, false, T>::run(w);
#pragma unroll
    for (int r = 0; r < F::R2; ++r) col[(j + F::R1 * r) * P] = w[r];  // X[j + R1 r], own slots
  }
  __syncthreads();
  // Green operator on the k-points (e, rho) of this tile: e strided over the Y*NC
  // threads of column t
  if (ok) {
    int k1, k2 = 0;
    if (D == 3) {
      k1 = (int)(rho / a.nh);
      k2 = (int)(rho - (long long)k1 * a.nh);
    } else {
      k1 = (int)rho;
    }
    const R x1 = a.xi1[k1], x2 = D == 3 ? a.xi2[k2] : R(0);
    T *tc = buf + t;
    for (int e = y + F::Y * z; e < M; e += F::Y * NC) {
      R xi[D];
      xi[0] = a.xi0[e];
      xi[1] = x1;
      if (D == 3) xi[D - 1] = x2;
      T f[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) f[c] = tc[e * P + c * Tt];
      if (!unit_xi<D>(xi, e, k1, k2, a.nyq0, a.nyq1, a.nyq2)) {
#pragma unroll
        for (int c = 0; c < NC; ++c) f[c] = T{R(0), R(0)};
      } else if (MODE == GM_FINITE) {
        green_finite_row<D>(f, xi, a.norm);
      } else {
        T o[NC];
        green_small<D>(f, o, xi, a.norm);
#pragma unroll
        for (int c = 0; c < NC; ++c) f[c] = o[c];
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) tc[e * P + c * Tt] = f[c];
    }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < F::NB; ++b) {
    const int j = y + F::Y * b;
    T w[F::R2];
#pragma unroll
    for (int r = 0; r < F::R2; ++r) w[r] = col[(j + F::R1 * r) * P];
    Dft<F::R2, true, T>::run(w);
#pragma unroll
    for (int r = 1; r < F::R2; ++r) w[r] = cmul(w[r], reg_tw<true>(tws, j * r));
#pragma unroll
    for (int r = 0; r < F::R2; ++r) col[(j + F::R1 * r) * P] = w[r];
  }
  __syncthreads();
  {
    T v[F::R1];
#pragma unroll
    for (int r = 0; r < F::R1; ++r) v[r] = col[(y * F::R1 + r) * P];
    Dft<F::R1, true, T>::run(v);
    if (ok) {
#pragma unroll
      for (int r = 0; r < F::R1; ++r) base[(y + F::Y * r) * se] = v[r];
    }
  }
}

}  // namespace musg
