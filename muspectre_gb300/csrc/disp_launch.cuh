// Host side of the displacement-space passes (disp.cuh): launch shapes, arguments and
// the dispatch over compile-time plans, shared by disp.cu and the passes' translation
// units (several, so that they build side by side).
#pragma once

#include <algorithm>
#include <vector>

#include "disp.cuh"
#include "launch_util.h"

namespace musg {

// FP32: axes with kernels of a compile-time plan.  The others' kernels hold a body per
// radix, compute strides and divide by lengths known at run time only, and spill where a
// radix above 12 does not fit their registers (160^3 small strain 382 -> 312 us an
// iteration, 63^3 70 -> 62 us, 45x77x81 76 -> 66 us, 16^3 54 -> 40 us).  16, multiples of 32 up
// to 256 and, in 3-D, the odd lengths of two factors up to 121: one kernel per length, pass
// and law is what a build of two minutes holds.  In FP64 the arithmetic, not the indexing,
// sets the pace.
#define MUSG_DISP_PLANS(X) \
  X(16, 4, 4) X(32, 8, 4) X(64, 8, 8) X(96, 12, 8) X(128, 16, 8) X(160, 16, 10) X(192, 16, 12) X(224, 16, 14) X(256, 16, 16)
#define MUSG_DISP_PLANS_ODD(X) \
  X(15, 5, 3) X(21, 7, 3) X(25, 5, 5) X(27, 9, 3) X(33, 11, 3) X(35, 7, 5) X(39, 13, 3) X(45, 9, 5) X(49, 7, 7) \
  X(51, 17, 3) X(55, 11, 5) X(63, 9, 7) X(65, 13, 5) X(75, 15, 5) X(77, 11, 7) X(81, 9, 9) X(85, 17, 5) X(91, 13, 7) \
  X(99, 11, 9) X(105, 15, 7) X(117, 13, 9) X(119, 17, 7) X(121, 11, 11)
inline int disp_fixed_plan(const TilePlan &pl) { return pl.blu ? 0 : pl.m; }

// launch shape of one pass
struct DispShape {
  int T = 0, G = 0, ntx = 0, nbx = 0, ng = 1, comps_at_once = 1, threads = 0, blocks = 0, sp = 0, S = 0;
  size_t smem = 0;
};

constexpr int kDispSms = 152;

inline bool disp_finite(const Spectral &sp) { return sp.proj_kind != MUSG_PROJ_SMALL_STRAIN; }

// Threads per block for tiles of P pencils: about 16 points of the tile per thread (one
// radix-16 or two radix-8 butterflies).  FP64, whose instructions take 16 cycles of an SM
// each: on grids too small to fill the SMs up to one butterfly per thread (35^3 149 ->
// 142 us an iteration; in FP32 the same rule cost more in per-thread setup than it
// gained, 63^3 77 -> 92 us).  A multiple of `unit` (the pencils of a pencil-fast tile, or
// a warp).
template <typename R> int disp_threads(const TilePlan &pl, long P, long blocks, long unit, long most) {
  const long tasks = P * (pl.r1 ? std::max(pl.r1, pl.r2) : pl.m / 4);
  const long fill = kDispSms * 1024L / std::max(1L, blocks);
  long t = P * pl.m / 16;
  if (sizeof(R) == 8) t = std::max(t, std::min(tasks, fill));
  t = std::max(64L, std::min(most, t));
  return (int)std::max(unit, std::min(most / unit, (t + unit - 1) / unit) * unit);
}
// Registers (kDispRegs): 512 threads of FP64 kernels fit, of their 2-D ones 384.  FP32: two
// blocks of 384 threads an SM; one of 480 left nothing to run at its barriers (160^3 small
// strain 422 -> 382 us an iteration).  Of the 2-D kernels' 128 registers two blocks of 256,
// where a grid has more blocks than SMs: 640^2 finite strain 75 -> 63 us, 613^2 327 -> 289.
template <typename R> long disp_most(const Spectral &sp, long blocks) {
  if (sizeof(R) == 8) return sp.g.dim == 3 ? 512 : 384;
  return sp.g.dim == 2 && blocks > kDispSms ? 256 : 384;
}
// registers of an iteration's kernel for the axis plan pl
template <typename R> int disp_regs(const Spectral &sp, const TilePlan &pl) {
  if (sizeof(R) == 4)
    switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, B) case M: return kDispRegs<R, 1>;
      MUSG_DISP_PLANS(MUSG_C)
#undef MUSG_C
      default: break;
    }
  return sp.g.dim == 2 ? kDispRegs<R, -2> : kDispRegs<R, 0>;
}
inline long lcm32(long p) {
  long a = p;
  while (a % 32) a += p;
  return a;
}

// axis-0 passes: tiles of T consecutive k-points.  16 complex values are a 128-byte
// line; narrower tiles where the grid would otherwise leave SMs without a block.  A
// Bluestein axis, several times the work per point, goes on below four points while most
// SMs have none (16 bytes at least, FP32 only below half a wave): 157 x 149 FP64, 38 blocks
// -> 150, 168 -> 109 ms; 359 x 324 small strain mixed, 41 -> 81, 12.8 -> 11.6 ms.  One
// point of 8 bytes costs more than it gains on half-filled grids (401^2 19.6 -> 20.5 ms).
template <typename R> DispShape disp_ax0_shape(const Spectral &sp, bool sums) {
  const bool fin = disp_finite(sp);
  const int D = sp.g.dim, na = fin ? 2 : D * (D + 1) / 2;
  const TilePlan &pl = sp.tile<R>(0);
  const long long Rr = disp_nk(sp) / sp.g.n[0];
  DispShape c;
  c.ng = fin ? D : 1;
  const long cb = 2 * (long)sizeof(R), per = (long)na * pl.m * cb * pl.buffers(), tw = pl.r1 ? pl.m * cb : 0;
  auto fits = [&](long T, long cap) { return T * per + tw <= cap; };
  long T = 16;
  while (T > 1 && !fits(T, 100 << 10)) T >>= 1;
  auto blocks = [&] { return (Rr + T - 1) / T * c.ng; };
  while (T > 4 && blocks() < 2 * kDispSms) T >>= 1;
  while (pl.blu && T > 1 && blocks() < (T * cb > 16 ? kDispSms : kDispSms / 2)) T >>= 1;
  if (!pl.m || !fits(T, optin_smem())) throw Error(MUSG_ERR_ARGUMENT, "first-axis FFT too long for one thread block");
  c.T = (int)T;
  c.ntx = (int)((Rr + T - 1) / T);
  c.smem = (size_t)(T * per + tw);
  auto threads = [&] {
    return disp_threads<R>(pl, na * T, (long)c.nbx * c.ng, lcm32(na * T), disp_most<R>(sp, (long)c.ntx * c.ng));
  };
  // With sums a block walks over several tiles, so that few sums are left to add up.  FP32:
  // as many blocks as are resident at once (128^3, 606 blocks of which 456 were resident:
  // 44 us, 456: 40 us, one block a tile: 45 us)
  c.nbx = c.ntx;
  if (sums) {
    c.threads = threads();
    const int regs = 65536 / (disp_regs<R>(sp, pl) * c.threads), mem = (int)((227l << 10) / (c.smem + 1024));
    const int resident = sizeof(R) == 8 ? 4 : std::max(1, std::min(8, std::min(regs, mem)));
    c.nbx = std::min(c.ntx, std::max(1, resident * kDispSms / c.ng));
  }
  c.blocks = c.nbx * c.ng;
  c.threads = threads();
  return c;
}

template <typename R> DispShape disp_mid_shape(const Spectral &sp) {
  const bool fin = disp_finite(sp);
  const TilePlan &pl = sp.tile<R>(1);
  DispShape c;
  c.ng = fin ? 3 : 6;
  c.comps_at_once = fin ? 3 : 1;
  const long cb = 2 * (long)sizeof(R), tw = pl.r1 ? pl.m * cb : 0, nh = disp_nh(sp);
  long per = (long)c.comps_at_once * pl.m * cb * pl.buffers();
  if (fin && per + tw > optin_smem()) {
    c.comps_at_once = 1;
    per = (long)pl.m * cb * pl.buffers();
  }
  if (!pl.m || per + tw > optin_smem()) throw Error(MUSG_ERR_ARGUMENT, "FFT axis too long for one thread block");
  long T = std::min<long>(fin ? 16 : 32, nh);
  while (T > 1 && T * per + tw > (56 << 10)) T = (T + 1) / 2;
  if (T * per + tw > optin_smem()) T = 1;
  while (T > 4 && (long long)c.ng * sp.g.n[0] * ((nh + T - 1) / T) < 2 * kDispSms) T = (T + 1) / 2;
  while (sizeof(R) == 8 && T > 1 && (long long)c.ng * sp.g.n[0] * ((nh + T - 1) / T) < kDispSms) T = (T + 1) / 2;
  const long nt = (nh + T - 1) / T;
  T = (nh + nt - 1) / nt;  // balanced: 65 -> 5 x 13
  c.T = (int)T;
  c.ntx = c.nbx = (int)nt;
  c.blocks = (int)((long long)c.ng * sp.g.n[0] * nt);
  c.smem = (size_t)(T * per + tw);
  c.threads = disp_threads<R>(pl, c.comps_at_once * T, c.blocks, c.comps_at_once * T, disp_most<R>(sp, c.blocks));
  return c;
}

// last-axis pass: pairs of rows of all components
template <typename R> DispShape disp_last_shape(const Spectral &sp) {
  const bool fin = disp_finite(sp);
  const int D = sp.g.dim, nl = fin ? D * D : D * (D + 1) / 2;
  const TilePlan &pl = sp.tile<R>(D - 1);
  DispShape c;
  const long cb = 2 * (long)sizeof(R), tw = pl.r1 ? pl.m * cb : 0;
  c.S = pl.r1;
  c.sp = pl.m;
  if (pl.r1) {
    const RowStrides r = row_strides(pl.r1, pl.r2);
    c.S = r.S;
    c.sp = r.sp;
  }
  long row = c.sp;
  if (sizeof(R) == 4) {  // a compile-time plan has its own strides
    switch (disp_fixed_plan(pl)) {
#define MUSG_C(M, A, B) \
  case M: row = std::max<long>(row, row_strides(A, B).sp); break;
      MUSG_DISP_PLANS(MUSG_C)
      MUSG_DISP_PLANS_ODD(MUSG_C)
#undef MUSG_C
      default: break;
    }
  }
  const long per = (long)nl * row * cb * pl.buffers();
  if (!pl.m || per + tw > optin_smem()) throw Error(MUSG_ERR_ARGUMENT, "last-axis FFT too long for one thread block");
  // rows until a block has about 160 threads, fewer where SMs would be without a block
  long g2 = std::max(1L, 160 * 16 / ((long)nl * pl.m));
  g2 = std::min<long>(g2, (sp.g.nrows + 1) / 2);
  while (g2 > 1 && g2 * per + tw > (64 << 10)) --g2;
  while (g2 > 1 && (sp.g.nrows + 2 * g2 - 1) / (2 * g2) < 2 * kDispSms) --g2;
  c.G = (int)(2 * g2);
  c.blocks = (int)((sp.g.nrows + c.G - 1) / c.G);
  c.smem = (size_t)(g2 * per + tw);
  c.threads = disp_threads<R>(pl, nl * g2, c.blocks, 16, disp_most<R>(sp, c.blocks));
  return c;
}

// arguments common to the passes
template <typename R> DispArgs<R> disp_base(Spectral &sp) {
  DispArgs<R> a{};
  const int D = sp.g.dim;
  a.n0 = sp.g.n[0];
  a.n1 = sp.g.n[1];
  a.nh = disp_nh(sp);
  a.L = sp.g.nlast();
  a.Rr = (int)(disp_nk(sp) / sp.g.n[0]);
  a.nk = disp_nk(sp);
  a.npx = sp.g.npx;
  a.nrows = sp.g.nrows;
  auto nyq = [&](int d) { return (sp.allow_even && sp.g.n[d] % 2 == 0) ? sp.g.n[d] / 2 : -1; };
  a.nyq0 = nyq(0);
  a.nyq1 = nyq(1);
  a.nyq2 = D == 3 ? nyq(2) : -1;
  a.scale = R(1.0 / std::sqrt((double)sp.g.npx));
  a.in_scale = 1.0;
  return a;
}
template <typename R> DispArgs<R> disp_with(DispArgs<R> a, const Spectral &sp, int axis, const DispShape &c) {
  const TilePlan &pl = sp.tile<R>(axis);
  a.ap = pl.device<R>();
  a.T = c.T;
  a.G = c.G;
  a.ntx = c.ntx;
  a.nbx = c.nbx;
  a.ng = c.ng;
  a.comps_at_once = c.comps_at_once;
  a.sp = c.sp;
  a.S = c.S;
  return a;
}

// one grouped launch: device tables of the problems' arguments and block prefix sums
template <typename R> struct DispGroup {
  const DispArgs<R> *tab = nullptr;
  const int *blk0 = nullptr;
  int B = 0;
};

template <typename R, typename K>
void disp_launch(K kernel, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
                 const DispGroup<R> *grp = nullptr) {
  allow_smem(kernel);
  launch_pdl(kernel, dim3(c.blocks, B), dim3(c.threads), c.smem, s, a, grp ? grp->tab : nullptr,
             grp ? grp->blk0 : nullptr, grp ? grp->B : 0);
  MUSG_CHECK_LAUNCH();
}

// runtime plans by dimension: radices up to 32 in 2-D (TileRun); of the FP64 grouped passes
// out of line in 3-D (build time).  The passes that run once per Newton step and per operator
// call have their stages inline like the iteration's: out of line they took two more
// shared-memory passes and barriers an axis (directional stiffness at 64^3 0.77 -> 0.71 ms,
// projection of 55^3 0.42 -> 0.40).
template <int D> constexpr int kRtPlan = D == 2 ? -2 : 0;
template <typename R, int D> constexpr int kGroupPlan = sizeof(R) == 4 || D == 2 ? kRtPlan<D> : -1;

// the passes: of an iteration (solo, batched, or grouped with grp), and the plain ones
template <typename R>
void disp_ax0_step(const Spectral &sp, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
                   const DispGroup<R> *grp);
template <typename R>
void disp_ax0_field(const Spectral &sp, bool from_x, const DispArgs<R> &a, const DispShape &c, cudaStream_t s);
template <typename R>
void disp_mid(const Spectral &sp, bool inv, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
              const DispGroup<R> *grp);
template <typename R>
void disp_ax0_dots(const Spectral &sp, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
                   const DispGroup<R> *grp);
template <typename R>
void disp_ax0_contract(const Spectral &sp, const DispArgs<R> &a, const DispShape &c, cudaStream_t s);
template <typename R, int D>
void disp_pixels(int tkind, const TilePlan &pl, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
                 const DispGroup<R> *grp);
// real field in (through the tangent, tkind TK_PLAIN: without it), spectrum out
template <typename R, int D>
void disp_pixels_in(bool fin, int tkind, bool delta, const DispArgs<R> &a, const DispShape &c, cudaStream_t s);
// spectrum in, real field out
template <typename R, int D>
void disp_pixels_out(bool fin, const DispArgs<R> &a, const DispShape &c, cudaStream_t s);

// FP32 3-D kernels of the odd compile-time plans (disp_odd_*.cu): false if the axis has none
bool disp_odd_ax0(bool fin, bool step, const TilePlan &, const DispArgs<float> &, const DispShape &, int B, cudaStream_t);
bool disp_odd_mid(bool fin, bool inv, const TilePlan &, const DispArgs<float> &, const DispShape &, int B, cudaStream_t);
bool disp_odd_pixels_finite(int tk, const TilePlan &, const DispArgs<float> &, const DispShape &, int B, cudaStream_t);
bool disp_odd_pixels_small(int tk, const TilePlan &, const DispArgs<float> &, const DispShape &, int B, cudaStream_t);

}  // namespace musg
