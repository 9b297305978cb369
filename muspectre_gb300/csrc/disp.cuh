// CG iteration in displacement space (device code), in FP64 (the plain method) and in FP32
// (the inner solve of the mixed method); the projection and the operator G(K:dF) of a
// general field run through the same passes.
//
// Every vector of the CG lies in the range of the projection G (the right-hand side is
// G(-P), x0 = 0), and a field in that range has D scalars per k-point instead of D^2:
//   finite strain  fhat_ij = v_i xi_j                      (xi the unit wave vector)
//   small strain   fhat_ij = (xi_i v_j + xi_j v_i) / 2
// So r, p, x and q = G(K:p) are stored as v: D complex values per half-spectrum point.
// With the unitary scaling 1/sqrt(N) the real-space inner product of two such fields is
// Parseval's sum with weight 2 on the points whose mirror image is not stored:
//   finite  sum_k w_k Re(conj(a) . b)
//   small   sum_k w_k Re(conj(a) . b + conj(a.xi) (b.xi)) / 2
// and the iteration of solver_cg.cc:76-97 runs on v with the same scalars alpha, beta.
// The Nyquist column of an even last axis is left out (the operator is zero there), so a
// row of 128 pixels is 64 complex values, a whole number of 128-byte lines.
// One iteration is five passes in 3-D and three in 2-D, R bytes per value:
//   ax0_inv   r += alpha q, x += alpha p, p = -r + beta p, then p's field along axis 0
//   mid_inv   axis 1 (3-D)
//   pixels    inverse along the last axis, tangent K:p per pixel, forward again: the
//             field is never stored in real space
//   mid_fwd   axis 1 (3-D)
//   ax0_fwd   axis 0, contraction with the wave vector = q, and the four sums p.q, r.q,
//             q.q, r.r
// Components on the way.  Small strain: the D (D + 1) / 2 entries i <= j.  Finite strain,
// one row i at a time: 3-D needs only two pencils along axis 0, k0 w and w (w = v/|k|),
// because the factors k1 and k2 of the other two columns commute with the axis-0
// transform; mid_inv expands w into the columns k1 w and k2 w, and mid_fwd contracts
// the two columns again.  2-D uses the columns k0 w, k1 w directly.
//
// Scalars.  ax0_fwd leaves per-block sums; the last of its (at most 8 x 152) blocks to
// finish adds them up in a fixed order and sets alpha, beta and the loop flag, once:
// the FP64 pipe is too slow to do it in every block of the next pass (2 us a block,
// 30 us of the 128^3 update pass).  alpha = r.r / p.q, and the new r.r for beta and the
// loop test is r.r + 2 alpha r.q + alpha^2 q.q, with r.r summed afresh in every
// iteration, so it does not drift; a drop below 1e-6 (FP32) of the old value, where that
// expression cancels, counts as 1e-6 (FP64 1e-14) and the next iteration's fresh r.r
// decides.
//
// Why: the real-space iteration this replaces moved 16 real fields and the tangent data
// (155 component spectra at 128^3 finite strain, 146 small strain) in eight launches;
// this one moves 101 and 78 in five.  One iteration on GB300, before -> now: 128^3 finite
// 291 -> 226 us, 63^3 115 -> 62, 45x77x81 164 -> 66, 160^3 small strain 1279 -> 309 (the
// odd and 5-smooth lengths also gain from the two-stage transforms of tile_fft.cuh).
// Of that at 128^3: without the Nyquist column (64 instead of 65 columns: whole lines)
// the axis-1 passes 39 -> 34 and 43 -> 33 us, sums in FP32 pairs 51 -> 45 us, the last
// axis by row pairs 88 -> 76 us.  What bounds the passes is latency between the barriers
// of a tile and instruction issue, at 20-24 warps an SM (80 registers), not bandwidth:
// 128^3 moves 850 MB in 226 us, 0.55 of the copy bandwidth.
// FP64 (bound by the FP64 pipe and, on small grids, latency): 51^2 252 -> 88 us, where
// the factors 17 x 3 replace Bluestein over 105, 35^3 182 -> 144; a 55^3 projection
// 2.05 -> 0.40 ms.
#pragma once

#include "spectral.cuh"
#include "tile_fft.cuh"

namespace musg {

// one problem's device pointers (a batched launch reads a table of them)
template <typename R> struct DispProb {
  typename V2<R>::T *spec;            // [ncomp][nk] work spectrum
  typename V2<R>::T *r, *q, *p, *x;   // [D][nk]
  CGState *st;
  double *partial;                    // 4 sums per block of ax0_fwd
  const R *xi0, *xi1, *xi2;           // wave numbers: equal grids may have boxes of different lengths
  TangentData<R> td;
};

template <typename R> struct DispArgs {
  TilePlanD<R> ap;        // the axis of this pass
  int n0, n1, nh, L;      // grid; nh: stored k-points of the last axis (disp_nh)
  int T, G;               // k-points per tile (strided axes), rows per tile (last axis)
  int ntx, nbx;           // tiles and blocks of a row group (component group)
  int ng;                 // row groups: D for the finite-strain axis passes
  int comps_at_once;      // mid passes, finite strain: 3, or 1 where a tile holds no more
  int nparts;             // blocks of ax0_fwd
  int sp, S;              // last-axis strides of pencils and slot groups
  int Rr;                 // k-points per e of axis 0 (a component holds fewer than 2^31)
  long long nk, npx, nrows;
  int nyq0, nyq1, nyq2;
  R scale;                // 1 / sqrt(N)
  const double *in64;     // real input planes
  double *in_prev;        // their previous values (IN_DELTA)
  double in_scale;
  R *out;                 // real output planes
  int tkind;              // tangent kind (TK_ANYFIN kernels)
  int gated;              // passes of an iteration run only while the state is active
  DispProb<R> pb;
  const DispProb<R> *tab;
  __device__ __forceinline__ void bind() {
    if (tab) pb = tab[blockIdx.y];
  }
};

// solo and batched launches take their arguments from the parameter (problem =
// blockIdx.y); grouped launches of different grids from a table, problem b owning the
// blocks [blk0[b], blk0[b+1])
template <bool GRP, typename R>
__device__ __forceinline__ DispArgs<R> disp_args(const DispArgs<R> &a0, const DispArgs<R> *gtab, const int *blk0, int B,
                                                 int &bid) {
  if constexpr (GRP) {
    const int b = group_problem(blk0, B);
    bid = (int)blockIdx.x - blk0[b];
    return gtab[b];
  } else {
    bid = (int)blockIdx.x;
    DispArgs<R> a = a0;
    a.bind();
    return a;
  }
}

template <typename R, int CR1, int CR2>
__device__ __forceinline__ void stage_tile_twiddles(typename V2<R>::T *dst, const TilePlanD<R> &pl) {
  if (CR1 <= 0 && pl.r1 == 0) return;  // three or more factors read them from global memory
  const int m = CR1 > 0 ? CR1 * CR2 : pl.m;
  for (int k = threadIdx.x; k < m; k += blockDim.x) dst[k] = pl.tw[k];
}

// registers per thread.  FP32: 80 for the runtime plans, whose radices above 12 would take
// up to 120 and halve the warps that hide the loads of all the others (they spill
// instead).  FP64 passes wait on the FP64 pipe, not on loads: 128.  2-D grids, whose
// radices go up to 32, are small: 128 and 168.
template <typename R, int CR1> constexpr int kDispRegs =
    sizeof(R) == 8 ? (CR1 == -2 ? 168 : 128) : CR1 == -2 ? 128 : 80;


// Sum of the threads' compensated accumulators over the block, by thread 0.  FP32: the
// warps add (sum, correction) pairs with Knuth's two-sum, an error of about 2^-46 in FP32
// instructions; FP64 shuffles and additions took 2 us a block on the slow FP64 pipe, all
// blocks at once at the end of the pass.
__device__ __forceinline__ void two_sum_add(Acc<float> &a, float s, float c) {
  const float t = a.s + s, z = t - a.s;
  a.c += ((a.s - (t - z)) + (s - z)) + c;
  a.s = t;
}
template <int N> __device__ __forceinline__ void block_sums(Acc<float> (&v)[N], double *out) {
  __shared__ float2 red[N][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float s = __shfl_down_sync(0xffffffffu, v[k].s, o), c = __shfl_down_sync(0xffffffffu, v[k].c, o);
      two_sum_add(v[k], s, c);
    }
  if (l == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) red[k][w] = make_float2(v[k].s, v[k].c);
  __syncthreads();
  if (threadIdx.x < N) {
    Acc<float> t;
    for (int i = 0; i < nw; ++i) two_sum_add(t, red[threadIdx.x][i].x, red[threadIdx.x][i].y);
    out[threadIdx.x] = t.value();
  }
}

__device__ __forceinline__ double disp_floor(float) { return 1e-6; }
__device__ __forceinline__ double disp_floor(double) { return 1e-14; }

template <int N> __device__ __forceinline__ void block_sums(Acc<double> (&v)[N], double *out) {
  __shared__ double red[N][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double s = v[k].s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (l == 0) red[k][w] = s;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double t = 0.0;
    for (int i = 0; i < nw; ++i) t += red[threadIdx.x][i];
    out[threadIdx.x] = t;
  }
}

// the end of an iteration, by the whole of its last block: the scalars from the nparts
// blocks' sums (p.q, r.q, q.q, r.r), and whether another iteration follows
// (solver_cg.cc:76-97).  The next update pass applies alpha and beta; without a further
// iteration it only finishes x.
template <typename R> __device__ __forceinline__ void disp_finish(CGState *st, const double *partial, int nparts) {
  // a quarter of the warps per sum, eight loads in flight per thread, added in index order
  __shared__ double red[4][8], total[4];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int k = w & 3, part = w >> 2, parts = max(1, nw >> 2);
  for (int kk = k; kk < 4 && part < parts; kk += min(nw, 4)) {  // fewer than four warps: several sums each
    double s = 0.0;
    for (int i = part * 32 + l; i < nparts; i += 8 * 32 * parts) {
      double t[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int q = i + u * 32 * parts;
        t[u] = q < nparts ? __ldcg(partial + (long long)4 * q + kk) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) s += t[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (l == 0) red[kk][part] = s;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int i = 0; i < parts; ++i) s += red[threadIdx.x][i];
    total[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double rr = total[3], alpha = rr / total[0];
    double rn = rr + 2.0 * alpha * total[1] + alpha * alpha * total[2];
    if (rn < disp_floor(R(0)) * rr) rn = disp_floor(R(0)) * rr;  // a NaN stays
    st->pAp = total[0];
    st->alpha = alpha;
    st->beta = rn / rr;
    rn += st->out2;
    st->rdr = rn;
    st->iter += 1;
    st->counter += 1;
    st->go = st->iter < st->maxiter && rn > st->tol2 ? 1 : 0;
    st->ticket = 0;
  }
}

// ------------------------------------------------------------ wave vectors
// component index of the work spectrum: finite strain keeps (i, j) at i + D j, small
// strain the entries (0,0) (1,1) [(2,2)] (0,1) [(0,2) (1,2)]
template <int D> struct Sym {
  static constexpr int N = D * (D + 1) / 2;
  __device__ static __forceinline__ constexpr int row(int s) { return s < D ? s : (D == 2 ? 0 : s == 5 ? 1 : 0); }
  __device__ static __forceinline__ constexpr int col(int s) { return s < D ? s : (D == 2 ? 1 : s == 3 ? 1 : 2); }
  __device__ static __forceinline__ constexpr int at(int i, int j) {
    return i == j ? i : (D == 2 ? 2 : 2 + i + j);  // (0,1) 3, (0,2) 4, (1,2) 5
  }
};
template <int D, bool FIN> struct DispComps {
  static constexpr int NA = FIN ? 2 : Sym<D>::N;      // pencils per k-point along axis 0 (a row of finite strain)
  static constexpr int ND = FIN ? 1 : D;              // unknowns per k-point of the block
  static constexpr int NL = FIN ? D * D : Sym<D>::N;  // components in real space
};

// wave numbers (not unit) of the points e of a k-point column (k1, k2) and 1/|k|; 0 where
// the operator is zero
template <int D, typename R> struct Wave {
  R k1, k2, s;
  int e_zero;  // the zero mode's e in this column, -1: none
  bool dead;
  int kl;      // index along the last axis
  __device__ __forceinline__ Wave(const DispArgs<R> &a, int rho) {
    int i1, i2 = 0;
    if (D == 3) i1 = FDiv(a.nh).div(rho, i2);
    else i1 = rho;
    k1 = a.pb.xi1[i1];
    k2 = D == 3 ? a.pb.xi2[i2] : R(0);
    s = k1 * k1;
    if (D == 3) s += k2 * k2;
    e_zero = i1 == 0 && i2 == 0 ? 0 : -1;
    dead = i1 == a.nyq1 || (D == 3 && i2 == a.nyq2);
    kl = D == 3 ? i2 : i1;
  }
  __device__ __forceinline__ R at(const DispArgs<R> &a, int e, R *k) const {
    k[0] = a.pb.xi0[e];
    k[1] = k1;
    if (D == 3) k[D - 1] = k2;
    if (dead || e == e_zero || e == a.nyq0) return R(0);
    return inv_sqrt(k[0] * k[0] + s);
  }
};

// ------------------------------------------------------------ axis 0, inverse
enum Ax0Mode : int {
  AX_STEP = 0,  // the CG update, then the field of p
  AX_X = 1,     // the field of x, in the units of the right-hand side
  AX_Q = 2      // the field of q
};

template <typename R, int D, bool FIN, int MODE, int CR1, int CR2, bool GRP>
__global__ void __maxnreg__((kDispRegs<R, CR1>)) k_ax0_inv(const DispArgs<R> a0, const DispArgs<R> *gtab, const int *blk0, int B) {
  using T = typename V2<R>::T;
  using C = DispComps<D, FIN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int bid;
  const DispArgs<R> a = disp_args<GRP, R>(a0, gtab, blk0, B, bid);
  const int Tt = a.T, n0 = CR1 > 0 ? CR1 * CR2 : a.n0;
  const int P = C::NA * Tt;
  T *buf = reinterpret_cast<T *>(smem_raw);
  T *buf2 = buf + (size_t)P * (CR1 > 0 ? CR1 * CR2 : a.ap.m);
  T *tws = (CR1 > 0 || a.ap.r1) ? buf2 : nullptr;
  stage_tile_twiddles<R, CR1, CR2>(tws, a.ap);
  const SlotMap<CR1, CR2> slots(a.ap, CR1 > 0 ? CR1 : a.ap.r1);
  const PencilMap map(P);
  const int g = bid / a.nbx, tile = bid - g * a.nbx;
  dep_wait();
  R alpha = R(0), beta = R(0);
  bool first = true, go = true;
  if (MODE == AX_STEP) {
    const CGState *st = a.pb.st;
    if (!st->active) return;
    first = st->iter == 0;
    go = st->go != 0;
    if (!first) {
      alpha = R(st->alpha);
      beta = R(st->beta);
    }
  }
  const R scale = MODE == AX_X ? a.scale * R(a.pb.st->xscale) : a.scale;
  // a thread keeps its k-point column t (T divides P, which divides the block)
  const int t = map.p % Tt, de = (int)blockDim.x / Tt;
  const int e0 = (int)threadIdx.x / Tt < de ? (int)threadIdx.x / Tt : kNoRow;
  const int rho = tile * Tt + t;
  const bool ok = rho < a.Rr;
  const Wave<D, R> wv(a, ok ? rho : 0);
  const long long ob = (long long)(FIN ? g : 0) * a.nk + rho;
  // independent loads of U points in flight before the first store
  constexpr int U = FIN ? 4 : 1;
  for (int eb = e0; eb < n0; eb += U * de) {
    T v[U][C::ND];
    if (MODE == AX_STEP) {
      T qv[U][C::ND], pv[U][C::ND], xv[U][C::ND];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = eb + u * de;
        const bool in = ok && e < n0;
#pragma unroll
        for (int d = 0; d < C::ND; ++d) {
          const long long o = ob + (long long)d * a.nk + e * a.Rr;
          v[u][d] = qv[u][d] = pv[u][d] = xv[u][d] = T{R(0), R(0)};
          if (in) {
            v[u][d] = a.pb.r[o];
            if (!first) {
              qv[u][d] = a.pb.q[o];
              pv[u][d] = a.pb.p[o];
              xv[u][d] = a.pb.x[o];
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = eb + u * de;
        const bool in = ok && e < n0;
#pragma unroll
        for (int d = 0; d < C::ND; ++d) {
          const long long o = ob + (long long)d * a.nk + e * a.Rr;
          const T x = T{xv[u][d].x + alpha * pv[u][d].x, xv[u][d].y + alpha * pv[u][d].y};
          const T r = T{v[u][d].x + alpha * qv[u][d].x, v[u][d].y + alpha * qv[u][d].y};
          v[u][d] = T{-r.x + beta * pv[u][d].x, -r.y + beta * pv[u][d].y};
          if (in && !first) {
            a.pb.x[o] = x;
            if (go) a.pb.r[o] = r;
          }
          if (in && go) a.pb.p[o] = v[u][d];
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = eb + u * de;
#pragma unroll
        for (int d = 0; d < C::ND; ++d) {
          const long long o = ob + (long long)d * a.nk + e * a.Rr;
          v[u][d] = ok && e < n0 ? (MODE == AX_X ? a.pb.x[o] : a.pb.q[o]) : T{R(0), R(0)};
        }
      }
    }
    if (!go) continue;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = eb + u * de;
      if (e >= n0) continue;
      R k[D];
      const R w = wv.at(a, e, k);
      const int s = slots.nat(e);
      if constexpr (FIN) {
        const R ws = w * scale, c0 = k[0] * ws, c1 = D == 3 ? ws : k[1] * ws;
        buf[map.at(s, t)] = T{c0 * v[u][0].x, c0 * v[u][0].y};
        buf[map.at(s, Tt + t)] = T{c1 * v[u][0].x, c1 * v[u][0].y};
      } else {
#pragma unroll
        for (int c = 0; c < C::NA; ++c) {
          const int i = Sym<D>::row(c), j = Sym<D>::col(c);
          const R f = R(0.5) * w * scale, ki = k[i] * f, kj = k[j] * f;
          buf[map.at(s, c * Tt + t)] = T{ki * v[u][j].x + kj * v[u][i].x, ki * v[u][j].y + kj * v[u][i].y};
        }
      }
    }
  }
  if (!go) return;
  __syncthreads();
  // this thread's pencil of the transform and where it goes
  const int c = map.p / Tt, comp = FIN ? g + D * c : c;
  T *out = a.pb.spec + (long long)comp * a.nk + rho;
  TileRun<CR1, CR2>::template io<true, R>(
      a.ap, map, buf, buf2, P, tws, [&](int, int s, int p) { return buf[map.at(s, p)]; },
      [&](int e, int, int, T v) {
        if (ok) out[e * a.Rr] = v;
      });
}

// ------------------------------------------------------------ axis 1 (3-D)
// spectrum [comp][k0][k1][k2].  Finite strain: block = (row i, k0, tile of k2), columns
// 0 (k0 w) and 1 (w) in, columns 0..2 out (INV), or the reverse contraction.  Columns
// run in descending order when a tile holds one at a time: the inverse reads w for
// column 2 before column 1 replaces it, the forward pass finds column 2's transform in
// memory when it forms column 1's.  Small strain: one component per block.
template <typename R, bool FIN, bool INV, int CR1, int CR2, bool GRP>
__global__ void __maxnreg__((kDispRegs<R, CR1>)) k_mid(const DispArgs<R> a0, const DispArgs<R> *gtab, const int *blk0, int B) {
  using T = typename V2<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int bid;
  const DispArgs<R> a = disp_args<GRP, R>(a0, gtab, blk0, B, bid);
  const int Tt = a.T, n1 = CR1 > 0 ? CR1 * CR2 : a.n1, nc = FIN ? a.comps_at_once : 1;
  const int P = nc * Tt;
  T *buf = reinterpret_cast<T *>(smem_raw);
  T *buf2 = buf + (size_t)P * (CR1 > 0 ? CR1 * CR2 : a.ap.m);
  T *tws = (CR1 > 0 || a.ap.r1) ? buf2 : nullptr;
  stage_tile_twiddles<R, CR1, CR2>(tws, a.ap);
  const SlotMap<CR1, CR2> slots(a.ap, CR1 > 0 ? CR1 : a.ap.r1);
  const PencilMap map(P);
  const int slab = bid / a.nbx, tile = bid - slab * a.nbx;  // slab: (row or component) * n0 + k0
  const int g = slab / a.n0, z = slab - g * a.n0;
  dep_wait();
  if (a.gated && !a.pb.st->go) return;
  const int t = map.p % Tt, k2 = tile * Tt + t;
  const bool ok = k2 < a.nh;
  const int nh = a.nh;
  const long long b = (long long)g * a.nk + (long long)z * n1 * nh + k2;
  __syncthreads();  // the twiddle copy
  if constexpr (!FIN) {
    T *base = a.pb.spec + b;
    TileRun<CR1, CR2>::template io<INV, R>(
        a.ap, map, buf, buf2, P, tws, [&](int e, int, int) { return ok ? base[e * nh] : T{R(0), R(0)}; },
        [&](int e, int, int, T v) {
          if (ok) base[e * nh] = v;
        });
  } else {
    T *b0 = a.pb.spec + b, *b1 = b0 + 3 * a.nk, *b2 = b1 + 3 * a.nk;
    const R x2 = ok ? a.pb.xi2[k2] : R(0);
    for (int hi = 2; hi >= 0; hi -= nc) {  // columns hi, hi - 1, ..., hi - nc + 1
      const int c0 = hi - nc + 1, c = c0 + map.p / Tt;  // this thread's column
      if (hi < 2) __syncthreads();                      // the previous column's tile is free
      if constexpr (INV) {
        // column 0: k0 w (from memory), 1: k1 w, 2: k2 w
        const T *src = c == 0 ? b0 : b1;
        T *dst = c == 0 ? b0 : c == 1 ? b1 : b2;
        const R kc = c == 0 ? R(1) : x2;
        auto ld = [&](int e, int, int) {
          const T w = ok ? src[e * nh] : T{R(0), R(0)};
          const R x1 = a.pb.xi1[e], k = c == 1 ? x1 : kc;
          return T{k * w.x, k * w.y};
        };
        auto st = [&](int e, int, int, T v) {
          if (ok) dst[e * nh] = v;
        };
        // columns 1 and 2 both read w, which column 1's stores replace: the barrier
        // between the stages stands between every read and the first store
        TileRun<CR1, CR2>::template io<true, R>(a.ap, map, buf, buf2, P, tws, ld, st);
      } else {
        const T *src = c == 0 ? b0 : c == 1 ? b1 : b2;
        const R k = c == 2 ? x2 : R(1);
        TileRun<CR1, CR2>::template io<false, R>(
            a.ap, map, buf, buf2, P, tws,
            [&](int e, int, int) {
              const T w = ok ? src[e * nh] : T{R(0), R(0)};
              return T{k * w.x, k * w.y};
            },
            [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; });
        __syncthreads();
        const int de = (int)blockDim.x / Tt;
        for (int e = (int)threadIdx.x / Tt; e < n1; e += de) {
          if (!ok || (int)threadIdx.x >= de * Tt) break;
          const int s = slots.nat(e);
          if (c0 == 0) b0[e * nh] = buf[map.at(s, t)];
          if (c0 <= 1 && hi >= 1) {
            const R k1 = a.pb.xi1[e];
            const T f1 = buf[map.at(s, (1 - c0) * Tt + t)];
            const T f2 = hi == 2 ? buf[map.at(s, (2 - c0) * Tt + t)] : b2[e * nh];
            b1[e * nh] = T{k1 * f1.x + f2.x, k1 * f1.y + f2.y};
          } else if (hi == 2) {
            b2[e * nh] = buf[map.at(s, t)];  // one at a time: column 2 waits for column 1
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------ axis 0, forward
enum Ax0Sums : int {
  AX_DOTS = 0,  // q and the sums p.q, r.q, q.q, r.r
  AX_OUT = 1    // q and its own q.q in the fourth sum
};

template <typename R, int D, bool FIN, int MODE, int CR1, int CR2, bool GRP>
__global__ void __maxnreg__((kDispRegs<R, CR1>)) k_ax0_fwd(const DispArgs<R> a0, const DispArgs<R> *gtab, const int *blk0, int B) {
  using T = typename V2<R>::T;
  using C = DispComps<D, FIN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int bid;
  const DispArgs<R> a = disp_args<GRP, R>(a0, gtab, blk0, B, bid);
  const int Tt = a.T, n0 = CR1 > 0 ? CR1 * CR2 : a.n0;
  const int P = C::NA * Tt;
  T *buf = reinterpret_cast<T *>(smem_raw);
  T *buf2 = buf + (size_t)P * (CR1 > 0 ? CR1 * CR2 : a.ap.m);
  T *tws = (CR1 > 0 || a.ap.r1) ? buf2 : nullptr;
  stage_tile_twiddles<R, CR1, CR2>(tws, a.ap);
  const SlotMap<CR1, CR2> slots(a.ap, CR1 > 0 ? CR1 : a.ap.r1);
  const PencilMap map(P);
  const int g = bid / a.nbx;
  const int t = map.p % Tt, c = map.p / Tt, comp = FIN ? g + D * c : c;
  const int de = (int)blockDim.x / Tt, e0 = (int)threadIdx.x / Tt < de ? (int)threadIdx.x / Tt : kNoRow;
  Acc<R> sum[4];
  dep_wait();
  if (a.gated && !a.pb.st->go) return;
  __syncthreads();  // the twiddle copy
  for (int tile = bid - g * a.nbx; tile < a.ntx; tile += a.nbx) {
    const int rho = tile * Tt + t;
    const bool ok = rho < a.Rr;
    const T *in = a.pb.spec + (long long)comp * a.nk + rho;
    TileRun<CR1, CR2>::template io<false, R>(
        a.ap, map, buf, buf2, P, tws, [&](int e, int, int) { return ok ? in[e * a.Rr] : T{R(0), R(0)}; },
        [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; });
    __syncthreads();
    const Wave<D, R> wv(a, ok ? rho : 0);
    const R wt = wv.kl == 0 ? R(1) : R(2);
    const long long ob = (long long)(FIN ? g : 0) * a.nk + rho;
    constexpr int U = FIN ? 4 : 2;
    for (int eb = e0; eb < n0; eb += U * de) {
      if (!ok) break;
      T pv[U][C::ND], rv[U][C::ND];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int d = 0; d < C::ND; ++d) {
          const int e = eb + u * de;
          const long long o = ob + (long long)d * a.nk + e * a.Rr;
          pv[u][d] = rv[u][d] = T{R(0), R(0)};
          if (MODE == AX_DOTS && e < n0) {
            pv[u][d] = a.pb.p[o];
            rv[u][d] = a.pb.r[o];
          }
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = eb + u * de;
        if (e >= n0) continue;
        R k[D];
        const R w = wv.at(a, e, k);
        const int s = slots.nat(e);
        T v[C::ND];
        if constexpr (FIN) {
          const T f0 = buf[map.at(s, t)], f1 = buf[map.at(s, Tt + t)];
          const R c1 = D == 3 ? R(1) : k[1], ws = w * a.scale;
          v[0] = T{(k[0] * f0.x + c1 * f1.x) * ws, (k[0] * f0.y + c1 * f1.y) * ws};
        } else {
#pragma unroll
          for (int d = 0; d < D; ++d) k[d] *= w;
          T f[C::NA];
#pragma unroll
          for (int q = 0; q < C::NA; ++q) f[q] = buf[map.at(s, q * Tt + t)];
          T tr[D], sc = T{R(0), R(0)};
#pragma unroll
          for (int i = 0; i < D; ++i) {
            tr[i] = T{R(0), R(0)};
#pragma unroll
            for (int j = 0; j < D; ++j) {
              const T h = f[Sym<D>::at(i < j ? i : j, i < j ? j : i)];
              tr[i].x += h.x * k[j];
              tr[i].y += h.y * k[j];
            }
            sc.x += tr[i].x * k[i];
            sc.y += tr[i].y * k[i];
          }
#pragma unroll
          for (int i = 0; i < D; ++i)
            v[i] = T{(R(2) * tr[i].x - sc.x * k[i]) * a.scale, (R(2) * tr[i].y - sc.y * k[i]) * a.scale};
        }
#pragma unroll
        for (int d = 0; d < C::ND; ++d) a.pb.q[ob + (long long)d * a.nk + e * a.Rr] = v[d];
        auto dot = [&](const T *x, const T *y) {
          R acc = R(0);
          if constexpr (FIN) {
            acc = x[0].x * y[0].x + x[0].y * y[0].y;
          } else {
            T ax = T{R(0), R(0)}, ay = T{R(0), R(0)};
#pragma unroll
            for (int d = 0; d < D; ++d) {
              acc += x[d].x * y[d].x + x[d].y * y[d].y;
              ax.x += x[d].x * k[d];
              ax.y += x[d].y * k[d];
              ay.x += y[d].x * k[d];
              ay.y += y[d].y * k[d];
            }
            acc = R(0.5) * (acc + ax.x * ay.x + ax.y * ay.y);
          }
          return wt * acc;
        };
        if (MODE == AX_DOTS) {
          sum[0].add(dot(pv[u], v));
          sum[1].add(dot(rv[u], v));
          sum[2].add(dot(v, v));
          sum[3].add(dot(rv[u], rv[u]));
        } else {
          sum[3].add(dot(v, v));
        }
      }
    }
    __syncthreads();  // the tile is free for the next one
  }
  if (a.pb.partial) block_sums(sum, a.pb.partial + 4 * (long long)bid);  // null: plain projections
  if (MODE == AX_DOTS && cg_last_block(a.pb.st, a.nparts)) disp_finish<R>(a.pb.st, a.pb.partial, a.nparts);
}

// ------------------------------------------------------------ last axis
enum PixIn : int {
  IN_SPEC = 0,   // inverse transform of the work spectrum
  IN_REAL = 1,   // in_scale * in64 (FP64 planes, all D^2 components)
  IN_DELTA = 2   // in_prev - in64, and in_prev = in64
};
enum PixOut : int { OUT_SPEC = 0, OUT_REAL = 1 };

template <int D, int TK, typename R>
__device__ __forceinline__ void pixel_tangent(const TangentData<R> &td, long long px, long long npx, const R *v, R *out) {
  TangentLocal<D, TK, R> tl;
  tl.load(td, px, npx);
  tl.apply(v, out);
}

// rows of G (pairs of rows share one complex transform) of all components; the pixels
// of the tile pass through shared memory once between the inverse and the forward
// transform, where the tangent is applied
template <typename R, int D, bool FIN, int TK, int IN, int OUT, int CR1, int CR2, bool GRP>
__global__ void __maxnreg__((kDispRegs<R, CR1>)) k_pixels(const DispArgs<R> a0, const DispArgs<R> *gtab, const int *blk0, int B) {
  using T = typename V2<R>::T;
  constexpr int NL = DispComps<D, FIN>::NL, D2 = D * D;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int bid;
  const DispArgs<R> a = disp_args<GRP, R>(a0, gtab, blk0, B, bid);
  const int L = CR1 > 0 ? CR1 * CR2 : a.L, H = (L + 1) / 2, G = a.G, G2 = G >> 1;
  const int P = NL * G2;
  const RowMap<CR1, CR2> lay(a.S, a.sp);
  T *buf = reinterpret_cast<T *>(smem_raw);
  T *buf2 = buf + (size_t)P * lay.sp;
  T *tws = (CR1 > 0 || a.ap.r1) ? buf2 : nullptr;
  stage_tile_twiddles<R, CR1, CR2>(tws, a.ap);
  const SlotMap<CR1, CR2> slots(a.ap, lay.S);
  const long long row0 = (long long)bid * G;
  dep_wait();
  if (a.gated) {
    CGState *st = a.pb.st;
    if (!st->go) {
      if (bid == 0 && threadIdx.x == 0) st->active = 0;  // the update pass before this one finished x
      return;
    }
  }
  T *cur = buf;
  // (row pair, k) of a load or store task; the components of a task follow each other
  const FDiv fH(H);
  auto task = [&](int idx, int &k) {
    if constexpr (CR1 > 0) {
      constexpr int h = (CR1 * CR2 + 1) / 2;
      k = idx % h;
      return idx / h;
    } else {
      return fH.div(idx, k);
    }
  };
  if (IN == IN_SPEC) {
    for (int idx = threadIdx.x; idx < G2 * H; idx += blockDim.x) {
      int k;
      const int g2 = task(idx, k);
      const long long rx = row0 + 2 * g2;
      const bool okx = rx < a.nrows, oky = rx + 1 < a.nrows;
      const T *src = a.pb.spec + rx * H + k;
      T X[NL], Y[NL];  // every load of the task in flight together
#pragma unroll
      for (int c = 0; c < NL; ++c) {
        X[c] = okx ? src[(long long)c * a.nk] : T{R(0), R(0)};
        Y[c] = oky ? src[(long long)c * a.nk + H] : T{R(0), R(0)};
      }
      const int pk = lay.at(slots.nat(k), g2), pm = lay.at(slots.nat(k > 0 ? L - k : L / 2), g2);
      const int pstep = G2 * lay.sp;
#pragma unroll
      for (int c = 0; c < NL; ++c) {
        T x = X[c], y = Y[c];
        if (k == 0) { x.y = R(0); y.y = R(0); }  // c2r uses the real part only
        buf[pk + c * pstep] = T{x.x - y.y, x.y + y.x};
        if (k > 0) buf[pm + c * pstep] = T{x.x + y.y, y.x - x.y};
        else if (L % 2 == 0) buf[pm + c * pstep] = T{R(0), R(0)};  // the Nyquist column is not stored: zero
      }
    }
    __syncthreads();
    cur = TileRun<CR1, CR2>::template run<true, R>(a.ap, lay, buf, buf2, P, tws);
  }
  // pixels: a thread takes the two rows of a pair at one e, the real and imaginary parts of
  // the pair's pencils
  const FDiv fL(L);
  for (int idx = threadIdx.x; idx < G2 * L; idx += blockDim.x) {
    int e, g2;
    if constexpr (CR1 > 0) {
      g2 = idx / (CR1 * CR2);
      e = idx % (CR1 * CR2);
    } else {
      g2 = fL.div(idx, e);
    }
    const long long px0 = (row0 + 2 * g2) * L + e;
    const int at0 = lay.at(slots.split(e), g2), pstep = G2 * lay.sp;
    T f[NL];
    if (IN == IN_SPEC)
#pragma unroll
      for (int c = 0; c < NL; ++c) f[c] = cur[at0 + c * pstep];
    auto pixel = [&](auto part, long long px, bool ok) {
      // part(c): the pixel's value of component c in f
      R v[D2], out[D2];
      constexpr bool kLocal = TK != TK_PLAIN && TK != TK_ANYFIN;
      TangentLocal<D, kLocal ? TK : TK_SMALL, R> tl;
      if constexpr (kLocal)
        if (ok) tl.load(a.pb.td, px, a.npx);
      if (IN == IN_SPEC) {
#pragma unroll
        for (int j = 0; j < D; ++j)
#pragma unroll
          for (int i = 0; i < D; ++i) v[i + D * j] = part(FIN ? i + D * j : Sym<D>::at(i < j ? i : j, i < j ? j : i));
      } else {
#pragma unroll
        for (int c = 0; c < D2; ++c) {
          const long long o = (long long)c * a.npx + px;
          v[c] = R(0);
          if (ok) {
            if (IN == IN_REAL) {
              v[c] = R(a.in_scale * a.in64[o]);
            } else {
              const double now = a.in64[o];
              v[c] = R(a.in_prev[o] - now);
              a.in_prev[o] = now;
            }
          }
        }
      }
      if constexpr (TK == TK_PLAIN) {
#pragma unroll
        for (int c = 0; c < D2; ++c) out[c] = v[c];
      } else {
#pragma unroll
        for (int c = 0; c < D2; ++c) out[c] = R(0);
        if (ok) {
          if constexpr (kLocal) {
            tl.apply(v, out);
          } else {
            switch (a.tkind) {
              case TK_FINITE: pixel_tangent<D, TK_FINITE>(a.pb.td, px, a.npx, v, out); break;
              case TK_KPRIME: pixel_tangent<D, TK_KPRIME>(a.pb.td, px, a.npx, v, out); break;
              case TK_MIXED: pixel_tangent<D, TK_MIXED>(a.pb.td, px, a.npx, v, out); break;
              case TK_FISO: pixel_tangent<D, TK_FISO>(a.pb.td, px, a.npx, v, out); break;
              case TK_GFINITE: pixel_tangent<D, TK_GFINITE>(a.pb.td, px, a.npx, v, out); break;
              default: pixel_tangent<D, TK_FULL>(a.pb.td, px, a.npx, v, out); break;
            }
          }
        }
      }
      if (OUT == OUT_REAL) {
        if (ok)
#pragma unroll
          for (int c = 0; c < D2; ++c) a.out[(long long)c * a.npx + px] = out[c];
      } else {
#pragma unroll
        for (int c = 0; c < NL; ++c) {
          if constexpr (FIN) {
            part(c) = out[c];
          } else {
            const int i = Sym<D>::row(c), j = Sym<D>::col(c);
            // a general input may be unsymmetric; the projection takes its symmetric part
            part(c) = (IN == IN_SPEC || i == j) ? out[i + D * j] : R(0.5) * (out[i + D * j] + out[j + D * i]);
          }
        }
      }
    };
    const long long row = row0 + 2 * g2;
    if constexpr (TK == TK_ANYFIN) {  // the kinds' code once, the parts swapped between
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        pixel([&](int c) -> R & { return f[c].x; }, px0 + h * L, row + h < a.nrows);
#pragma unroll
        for (int c = 0; c < NL; ++c) f[c] = T{f[c].y, f[c].x};
      }
    } else {
      pixel([&](int c) -> R & { return f[c].x; }, px0, row < a.nrows);
      pixel([&](int c) -> R & { return f[c].y; }, px0 + L, row + 1 < a.nrows);
    }
    if (OUT == OUT_SPEC)
#pragma unroll
      for (int c = 0; c < NL; ++c) cur[at0 + c * pstep] = f[c];
  }
  if (OUT == OUT_REAL) return;
  __syncthreads();
  const T *res = TileRun<CR1, CR2>::template run<false, R>(a.ap, lay, cur, cur == buf ? buf2 : buf, P, tws);
  // unpack the two real spectra: X = (Z_k + conj Z_{L-k})/2, Y = -i (Z_k - conj Z_{L-k})/2
  for (int idx = threadIdx.x; idx < G2 * H; idx += blockDim.x) {
    int k;
    const int g2 = task(idx, k);
    const long long rx = row0 + 2 * g2;
    const bool okx = rx < a.nrows, oky = rx + 1 < a.nrows;
    T *dst = a.pb.spec + rx * H + k;
    const int pk = lay.at(slots.nat(k), g2), pm = lay.at(slots.nat(k == 0 ? 0 : L - k), g2), pstep = G2 * lay.sp;
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const T z = res[pk + c * pstep], zn = res[pm + c * pstep];
      if (okx) dst[(long long)c * a.nk] = T{R(0.5) * (z.x + zn.x), R(0.5) * (z.y - zn.y)};
      if (oky) dst[(long long)c * a.nk + H] = T{R(0.5) * (z.y + zn.y), R(-0.5) * (z.x - zn.x)};
    }
  }
}

}  // namespace musg
