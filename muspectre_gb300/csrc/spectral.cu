// The FFT engine's transforms (FP64): launchers of the passes of spectral.cuh.
#include <algorithm>

#include "launch_util.h"
#include "spectral.cuh"

namespace musg {

namespace {

struct Cfg {
  int per;       // rows per block (last pass) or tile (axis / green passes)
  int blocks;
  size_t smem;
  int threads;
};


// shared memory per block: two ping-pong buffers of (pencils x m) complex values
template <typename R> Cfg last_cfg(const Spectral &sp) {
  const AxisPlan &ap = sp.ax[sp.g.dim - 1];
  const long per_pair = (long)sp.ncomp * ap.m;
  const long eb = 2 * sizeof(typename V2<R>::T);
  const long target = kEngineBytes[0];
  long g2 = std::min(std::max(1L, target / (per_pair * eb)), (long)optin_smem() / (per_pair * eb));
  if (g2 < 1) throw Error(MUSG_ERR_ARGUMENT, "last-axis FFT too long for one thread block");
  g2 = std::min<long>(g2, 16);
  g2 = std::min<long>(g2, (sp.g.nrows + 1) / 2);
  Cfg c;
  c.per = (int)(2 * g2);
  c.blocks = (int)((sp.g.nrows + c.per - 1) / c.per);
  c.smem = (size_t)(g2 * per_pair * eb);
  c.threads = kEngineThreads[0];
  return c;
}

template <typename R> Cfg axis_cfg(const Spectral &sp, int axis, long long inner, long long nbatch) {
  const AxisPlan &ap = sp.ax[axis];
  const long eb = 2 * sizeof(typename V2<R>::T);
  const long target = kEngineBytes[1];
  long T = std::min(std::max(1L, target / (ap.m * eb)), (long)optin_smem() / (ap.m * eb));
  if (T < 1) throw Error(MUSG_ERR_ARGUMENT, "FFT axis too long for one thread block");
  T = std::min<long>(T, 32);
  T = std::min<long>(T, inner);
  // balance the tiles over the inner extent (65 -> 22 + 22 + 21, not 32 + 32 + 1)
  const long nt = (inner + T - 1) / T;
  T = (inner + nt - 1) / nt;
  Cfg c;
  c.per = (int)T;
  const long long ntiles = (inner + T - 1) / T;
  c.blocks = (int)(ntiles * nbatch);
  c.smem = (size_t)(T * ap.m * eb);
  c.threads = kEngineThreads[1];
  return c;
}

template <typename R> Cfg green_cfg(const Spectral &sp, long long Rr) {
  const AxisPlan &ap = sp.ax[0];
  const long per = (long)sp.ncomp * ap.m;
  const long eb = 2 * sizeof(typename V2<R>::T);
  const long target = kEngineBytes[2];
  long T = std::min(std::max(1L, target / (per * eb)), (long)optin_smem() / (per * eb));
  if (T < 1) throw Error(MUSG_ERR_ARGUMENT, "first-axis FFT too long for one thread block");
  T = std::min<long>(T, 32);
  T = std::min<long>(T, Rr);
  Cfg c;
  c.per = (int)T;
  c.blocks = (int)((Rr + T - 1) / T);
  c.smem = (size_t)(T * per * eb);
  c.threads = kEngineThreads[2];
  return c;
}

template <typename R> typename V2<R>::T *spec_of(Spectral &sp);
template <> double2 *spec_of<double>(Spectral &sp) { return (double2 *)sp.spec64; }
template <typename R> LastArgs<R> last_args(Spectral &sp, const Cfg &c) {
  LastArgs<R> a{};
  a.ap = sp.ax[sp.g.dim - 1].device<R>();
  a.L = sp.g.nlast();
  a.H = sp.g.nh;
  a.G = c.per;
  a.ncomp = sp.ncomp;
  a.nrows = sp.g.nrows;
  a.npx = sp.g.npx;
  a.nk = sp.g.nk;
  a.spec = spec_of<R>(sp);
  return a;
}

template <typename R> void run_axis(Spectral &sp, bool inv, cudaStream_t s) {
  // 3-D only: pencils along axis 1 of [c][k0][k1][k2h]
  const long long inner = sp.g.nh;
  const Cfg c = axis_cfg<R>(sp, 1, inner, (long long)sp.ncomp * sp.g.n[0]);
  AxisArgs<R> a{};
  a.ap = sp.ax[1].device<R>();
  a.nax = sp.g.n[1];
  a.T = c.per;
  a.ntiles = (int)((inner + c.per - 1) / c.per);
  a.se = sp.g.nh;
  a.inner = inner;
  a.sb = (long long)sp.g.n[1] * sp.g.nh;
  a.spec = spec_of<R>(sp);
  auto k = inv ? k_axis<R, true> : k_axis<R, false>;
  allow_smem(k);
  launch_pdl(k, dim3(c.blocks), dim3(c.threads), c.smem, s, a);
  MUSG_CHECK_LAUNCH();
}

template <typename R> void run_first(Spectral &sp, bool inv, cudaStream_t s) {
  const long long Rr = sp.g.nk / sp.g.n[0];
  const Cfg c = green_cfg<R>(sp, Rr);
  GreenArgs<R> a{};
  a.ap = sp.ax[0].device<R>();
  a.n0 = sp.g.n[0];
  a.T = c.per;
  a.ncomp = sp.ncomp;
  a.Rr = Rr;
  a.nk = sp.g.nk;
  a.spec = spec_of<R>(sp);
  auto k = inv ? k_green<R, GM_INV> : k_green<R, GM_FWD>;
  allow_smem(k);
  launch_pdl(k, dim3(c.blocks), dim3(c.threads), c.smem, s, a);
  MUSG_CHECK_LAUNCH();
}

}  // namespace

template <typename R>
void spectral_forward(Spectral &sp, const R *in, R scale, cudaStream_t s) {
  const Cfg c = last_cfg<R>(sp);
  LastArgs<R> a = last_args<R>(sp, c);
  a.in = in;
  a.scale = scale;
  auto k = k_last_fwd<R>;
  allow_smem(k);
  launch_pdl(k, dim3(c.blocks), dim3(c.threads), c.smem, s, a);
  MUSG_CHECK_LAUNCH();
  if (sp.g.dim == 3) run_axis<R>(sp, false, s);
  run_first<R>(sp, false, s);
}

template <typename R>
void spectral_inverse(Spectral &sp, R *out, R scale, cudaStream_t s) {
  run_first<R>(sp, true, s);
  if (sp.g.dim == 3) run_axis<R>(sp, true, s);
  const Cfg c = last_cfg<R>(sp);
  LastArgs<R> a = last_args<R>(sp, c);
  a.out = out;
  a.scale = scale;
  auto k = k_last_inv<R>;
  allow_smem(k);
  launch_pdl(k, dim3(c.blocks), dim3(c.threads), c.smem, s, a);
  MUSG_CHECK_LAUNCH();
}

template void spectral_forward<double>(Spectral &, const double *, double, cudaStream_t);
template void spectral_inverse<double>(Spectral &, double *, double, cudaStream_t);

}  // namespace musg
