// The displacement-space CG (disp.cuh): iterations, projections and batches from its passes.
#include <cstring>
#include <memory>

#include "disp_launch.cuh"

namespace musg {
namespace {

// the five passes' shapes and arguments of one grid
template <typename R> struct DispPasses {
  DispShape ci, cf, cm, cl;       // axis 0 inverse and forward, axis 1, last axis
  DispArgs<R> ai, af, am, al;
};
template <typename R> DispPasses<R> disp_passes(Spectral &sp, const DispProb<R> &pb) {
  DispPasses<R> p;
  const int D = sp.g.dim;
  p.ci = disp_ax0_shape<R>(sp, false);
  p.cf = disp_ax0_shape<R>(sp, true);
  p.cl = disp_last_shape<R>(sp);
  DispArgs<R> a = disp_base<R>(sp);
  a.pb = pb;
  a.nparts = p.cf.blocks;
  a.gated = 1;
  p.ai = disp_with<R>(a, sp, 0, p.ci);
  p.af = disp_with<R>(a, sp, 0, p.cf);
  p.al = disp_with<R>(a, sp, D - 1, p.cl);
  if (D == 3) {
    p.cm = disp_mid_shape<R>(sp);
    p.am = disp_with<R>(a, sp, 1, p.cm);
  }
  return p;
}

// The solve runs on the right-hand side scaled to unit norm: q.q grows with the square of
// the stiffness and would leave the range of FP32 for residuals in Pa.  x is scaled back
// when it is read (AX_X).
__global__ void k_disp_start(CGState *st, const double *out2, const double *range2, double tol, int maxiter) {
  const double in = *range2, out = out2 ? *out2 : 0.0;
  st->xscale = sqrt(in);
  st->out2 = out / in;
  st->rdr = st->rhs_norm2 = (in + out) / in;
  st->tol2 = tol * tol * st->rhs_norm2;
  st->alpha = st->beta = st->pAp = 0.0;
  st->iter = 0;
  st->maxiter = maxiter;
  st->ticket = 0;
  // solver_cg.cc:76-77: the first iteration is forced
  st->active = st->go = maxiter > 0 ? 1 : 0;
}

// r = -b (over the scale), x = 0.  The points of the plane k_last = 0 come in pairs (k, -k)
// of one real field; rounding leaves b unsymmetric there, the operator's inverse transform
// drops that part and no iteration could reduce it, so each pair takes its mean (in a
// residual accumulated over Newton steps the rounding is that of the largest one, and
// the CG stalled on it).
template <typename R>
__global__ void k_disp_init(const typename V2<R>::T *__restrict__ b, typename V2<R>::T *__restrict__ r,
                            typename V2<R>::T *__restrict__ x, int D, int n0, int n1, int nh, const CGState *st) {
  using T = typename V2<R>::T;
  const R c = (R)(-1.0 / st->xscale);
  const unsigned rows = (unsigned)D * n0 * n1, n = rows * (unsigned)nh;  // n1: 1 in 2-D
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    T v = b[i];
    if (i % nh == 0) {
      const unsigned row = i / nh, k1 = row % n1, dk0 = row / n1, k0 = dk0 % n0;
      const unsigned m0 = k0 ? n0 - k0 : 0, m1 = k1 ? n1 - k1 : 0;
      const T w = b[((size_t)(dk0 - k0 + m0) * n1 + m1) * nh];
      v = T{R(0.5) * (v.x - w.x), R(0.5) * (v.y + w.y)};  // xi is odd: v(-k) = -conj v(k)
    }
    r[i] = T{c * v.x, c * v.y};
    x[i] = T{R(0), R(0)};
  }
}

// the fourth sums of the blocks, in a fixed order
__global__ void k_disp_sum(const double *partial, int nparts, double *out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += partial[4 * i + 3];
  s = block_sum(s);
  if (threadIdx.x == 0) *out = s;
}

__global__ void k_disp_convert(const double2 *__restrict__ a, float2 *__restrict__ b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double2 v = a[i];
    b[i] = make_float2((float)v.x, (float)v.y);
  }
}

// The residual of the mixed method: r64 += change (the FP32 projection of the stress change,
// in r32), r32 = r64 rounded, and a block's part of |r64|^2 in FP64 (Parseval's sum of the
// header of disp.cuh) where k_disp_sum reads it.  Bound by its 48 bytes a complex value, 151 MB
// at 128^3, and on small grids by its launch; once per residual after the second of a load
// step: 32^3 elasto-plastic, some hundred of them, 97.9 -> 99.6 ms a solve, 128^3 spheres 38.4
// ms before and after.
template <int D, bool FIN>
__global__ void k_disp_add(double2 *__restrict__ r64, float2 *__restrict__ r32, const DispArgs<double> a, double *partial) {
  double sum = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.nk; i += (long long)gridDim.x * blockDim.x) {
    double2 v[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const long long o = (long long)d * a.nk + i;
      const float2 c = r32[o];
      v[d] = r64[o];
      v[d].x += (double)c.x;
      v[d].y += (double)c.y;
      r64[o] = v[d];
      r32[o] = make_float2((float)v[d].x, (float)v[d].y);
    }
    const int e = (int)(i / a.Rr), rho = (int)(i - (long long)e * a.Rr);
    const Wave<D, double> wv(a, rho);
    double acc = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) acc += v[d].x * v[d].x + v[d].y * v[d].y;
    if constexpr (!FIN) {
      double k[D], lx = 0.0, ly = 0.0;
      const double w = wv.at(a, e, k);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        lx += v[d].x * k[d] * w;
        ly += v[d].y * k[d] * w;
      }
      acc = 0.5 * (acc + lx * lx + ly * ly);
    }
    sum += wv.kl == 0 ? acc : 2.0 * acc;
  }
  sum = block_sum(sum);
  if (threadIdx.x == 0) partial[4 * blockIdx.x + 3] = sum;
}

template <typename R> typename V2<R>::T *work_spectrum(Spectral &sp);
template <> double2 *work_spectrum<double>(Spectral &sp) {
  sp.ensure_tiles();
  return (double2 *)sp.spec64;
}
template <> float2 *work_spectrum<float>(Spectral &sp) {
  sp.ensure32();
  return (float2 *)sp.spec32;
}

template <typename R> DispProb<R> disp_prob(Spectral &sp, const DispVectors &v, CGState *st, double *partial) {
  using T = typename V2<R>::T;
  DispProb<R> pb;
  pb.spec = work_spectrum<R>(sp);
  pb.r = (T *)v.r;
  pb.q = (T *)v.q;
  pb.p = (T *)v.p;
  pb.x = (T *)v.x;
  pb.st = st;
  pb.partial = partial;
  pb.xi0 = xi_table<R>(sp, 0);
  pb.xi1 = xi_table<R>(sp, 1);
  pb.xi2 = sp.g.dim == 3 ? xi_table<R>(sp, 2) : nullptr;
  return pb;
}

template <typename R>
void pixels(const Spectral &sp, int tkind, const DispArgs<R> &a, const DispShape &c, int B, cudaStream_t s,
            const DispGroup<R> *grp) {
  if (sp.g.dim == 2) disp_pixels<R, 2>(tkind, sp.tile<R>(1), a, c, B, s, grp);
  else disp_pixels<R, 3>(tkind, sp.tile<R>(2), a, c, B, s, grp);
}

// q (the vectors' q) -> real planes, ungated
template <typename R> void inverse_from(Spectral &sp, DispProb<R> pb, bool from_x, R *out, cudaStream_t s) {
  DispPasses<R> p = disp_passes<R>(sp, pb);
  p.ai.gated = p.am.gated = p.al.gated = 0;
  p.al.out = out;
  const bool fin = disp_finite(sp);
  disp_ax0_field<R>(sp, from_x, p.ai, p.ci, s);
  if (sp.g.dim == 3) disp_mid<R>(sp, true, p.am, p.cm, 1, s, nullptr);
  if (sp.g.dim == 2) disp_pixels_out<R, 2>(fin, p.al, p.cl, s);
  else disp_pixels_out<R, 3>(fin, p.al, p.cl, s);
}

// real planes (through the tangent unless tkind is TK_PLAIN) -> q, its q.q in *sum2
template <typename R>
void forward_to(Spectral &sp, DispProb<R> pb, int tkind, const double *in, double *prev, double in_scale, double *sum2,
                cudaStream_t s) {
  DispPasses<R> p = disp_passes<R>(sp, pb);
  p.af.gated = p.am.gated = p.al.gated = 0;
  p.al.in64 = in;
  p.al.in_prev = prev;
  p.al.in_scale = in_scale;
  const bool fin = disp_finite(sp);
  if (sp.g.dim == 2) disp_pixels_in<R, 2>(fin, tkind, prev != nullptr, p.al, p.cl, s);
  else disp_pixels_in<R, 3>(fin, tkind, prev != nullptr, p.al, p.cl, s);
  if (sp.g.dim == 3) disp_mid<R>(sp, false, p.am, p.cm, 1, s, nullptr);
  disp_ax0_contract<R>(sp, p.af, p.cf, s);
  if (sum2) {
    k_disp_sum<<<1, 256, 0, s>>>(pb.partial, p.cf.blocks, sum2);
    MUSG_CHECK_LAUNCH();
  }
}

}  // namespace

template <typename R>
void disp_residual(Spectral &sp, int tkind, const TangentData<R> &td, void *rhat, const double *field, double *prev,
                   double scale, double *partial, double *norm2, cudaStream_t s) {
  DispVectors v;
  v.q = rhat;
  DispProb<R> pb = disp_prob<R>(sp, v, nullptr, partial);
  pb.td = td;
  forward_to<R>(sp, pb, tkind, field, prev, scale, norm2, s);
}

template <typename R>
void disp_start(Spectral &sp, const DispVectors &v, const void *rhat, CGState *st, double tol, int maxiter,
                const double *out2, const double *range2, cudaStream_t s) {
  using T = typename V2<R>::T;
  const long long n = disp_nk(sp) * sp.g.dim;
  if (n > 0xf0000000ll) throw Error(MUSG_ERR_ARGUMENT, "grid too large for the CG solver");
  k_disp_start<<<1, 1, 0, s>>>(st, out2, range2, tol, maxiter);
  MUSG_CHECK_LAUNCH();
  k_disp_init<R><<<reduce_blocks(n), 256, 0, s>>>((const T *)rhat, (T *)v.r, (T *)v.x, sp.g.dim, sp.g.n[0],
                                                  sp.g.dim == 3 ? sp.g.n[1] : 1, disp_nh(sp), st);
  MUSG_CHECK_LAUNCH();
}

template <typename R>
void disp_iteration(Spectral &sp, int tkind, const TangentData<R> &td, const DispVectors &v, CGState *st,
                    double *partial, cudaStream_t s, cudaEvent_t *ev) {
  DispProb<R> pb = disp_prob<R>(sp, v, st, partial);
  pb.td = td;
  const DispPasses<R> p = disp_passes<R>(sp, pb);
  int k = 0;
  auto mark = [&]() {
    if (ev) MUSG_CUDA(cudaEventRecord(ev[k++], s));
  };
  mark();
  disp_ax0_step<R>(sp, p.ai, p.ci, 1, s, nullptr);
  mark();
  if (sp.g.dim == 3) {
    disp_mid<R>(sp, true, p.am, p.cm, 1, s, nullptr);
    mark();
  }
  pixels<R>(sp, tkind, p.al, p.cl, 1, s, nullptr);
  mark();
  if (sp.g.dim == 3) {
    disp_mid<R>(sp, false, p.am, p.cm, 1, s, nullptr);
    mark();
  }
  disp_ax0_dots<R>(sp, p.af, p.cf, 1, s, nullptr);
  mark();
}

template <typename R>
void disp_solution(Spectral &sp, const DispVectors &v, CGState *st, R *x, cudaStream_t s) {
  inverse_from<R>(sp, disp_prob<R>(sp, v, st, nullptr), true, x, s);
}

template <typename R>
void disp_operator(Spectral &sp, int tkind, const TangentData<R> &td, const double *in, R *out, cudaStream_t s) {
  // q in the work spectrum itself: a block of the contraction has read its tile's
  // components before it writes q over the first ones, and the inverse likewise
  DispVectors v;
  v.q = work_spectrum<R>(sp);
  DispProb<R> pb = disp_prob<R>(sp, v, nullptr, nullptr);
  pb.td = td;
  forward_to<R>(sp, pb, tkind, in, nullptr, 1.0, nullptr, s);
  inverse_from<R>(sp, pb, false, out, s);
}

template <typename R> void disp_field(Spectral &sp, void *qhat, R *out, cudaStream_t s) {
  DispVectors v;
  v.q = qhat;
  inverse_from<R>(sp, disp_prob<R>(sp, v, nullptr, nullptr), false, out, s);
}

void disp_convert(const Spectral &sp, const void *v64, void *v32, cudaStream_t s) {
  const long long n = disp_nk(sp) * sp.g.dim;
  k_disp_convert<<<reduce_blocks(n), 256, 0, s>>>((const double2 *)v64, (float2 *)v32, n);
  MUSG_CHECK_LAUNCH();
}

void disp_accumulate(Spectral &sp, void *r64, void *r32, double *partial, double *norm2, cudaStream_t s) {
  DispProb<double> pb{};
  pb.xi0 = xi_table<double>(sp, 0);
  pb.xi1 = xi_table<double>(sp, 1);
  pb.xi2 = sp.g.dim == 3 ? xi_table<double>(sp, 2) : nullptr;
  DispArgs<double> a = disp_base<double>(sp);
  a.pb = pb;
  const int nb = reduce_blocks(a.nk);
  const bool fin = disp_finite(sp);
  auto *k = sp.g.dim == 2 ? (fin ? k_disp_add<2, true> : k_disp_add<2, false>)
                          : (fin ? k_disp_add<3, true> : k_disp_add<3, false>);
  k<<<nb, 256, 0, s>>>((double2 *)r64, (float2 *)r32, a, partial);
  MUSG_CHECK_LAUNCH();
  k_disp_sum<<<1, 256, 0, s>>>(partial, nb, norm2);
  MUSG_CHECK_LAUNCH();
}

#define MUSG_INSTANTIATE_DISP(R)                                                                                      \
  template void disp_residual<R>(Spectral &, int, const TangentData<R> &, void *, const double *, double *, double,   \
                                 double *, double *, cudaStream_t);                                                   \
  template void disp_start<R>(Spectral &, const DispVectors &, const void *, CGState *, double, int, const double *,  \
                              const double *, cudaStream_t);                                                          \
  template void disp_iteration<R>(Spectral &, int, const TangentData<R> &, const DispVectors &, CGState *, double *,  \
                                  cudaStream_t, cudaEvent_t *);                                                       \
  template void disp_solution<R>(Spectral &, const DispVectors &, CGState *, R *, cudaStream_t);                      \
  template void disp_field<R>(Spectral &, void *, R *, cudaStream_t);                                                 \
  template void disp_operator<R>(Spectral &, int, const TangentData<R> &, const double *, R *, cudaStream_t);
MUSG_INSTANTIATE_DISP(float)
MUSG_INSTANTIATE_DISP(double)

// ------------------------------------------------------------------ batches
// problems of one grid: a device table indexed by blockIdx.y; of different grids: per
// pass a table of arguments and the prefix sums of the problems' blocks
struct DispBatch {
  virtual ~DispBatch() {}
  virtual void run(cudaStream_t s) = 0;
};

namespace {

template <typename T> void upload(DevBuf &d, const std::vector<T> &v) {
  d.alloc(v.size() * sizeof(T));
  MUSG_CUDA(cudaMemcpy(d.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
}

template <typename R> struct DispBatchR : DispBatch {
  bool uniform = true;
  int B = 0, dim = 0, tkind = 0;
  Spectral *sp0 = nullptr;
  DispPasses<R> p;                  // uniform: the shared shapes; else the launches' sizes
  DevBuf tab, gi, gm, gl, gf, blk;  // tables; blk: four prefix sums of B + 1

  DispBatchR(const std::vector<DispProblem> &probs, int tkind_, bool uniform_)
      : uniform(uniform_), B((int)probs.size()), dim(probs[0].sp->g.dim), tkind(tkind_), sp0(probs[0].sp) {
    std::vector<DispProb<R>> tb;
    for (const DispProblem &q : probs) {
      DispProb<R> pb = disp_prob<R>(*q.sp, q.v, q.st, q.partial);
      if constexpr (sizeof(R) == 4) pb.td = q.td32;
      else pb.td = q.td64;
      tb.push_back(pb);
    }
    if (uniform) {
      upload(tab, tb);
      p = disp_passes<R>(*sp0, DispProb<R>{});
      for (DispArgs<R> *a : {&p.ai, &p.am, &p.al, &p.af}) a->tab = tab.as<DispProb<R>>();
      return;
    }
    const int n = B + 1;
    std::vector<DispArgs<R>> vi, vm, vl, vf;
    std::vector<int> bk(4 * n, 0);
    for (int k = 0; k < B; ++k) {
      Spectral &sp = *probs[k].sp;
      if (sp.g.dim != dim || disp_finite(sp) != disp_finite(*sp0))
        throw Error(MUSG_ERR_ARGUMENT, "a grouped operator needs one dimension, projection and component count");
      const DispPasses<R> q = disp_passes<R>(sp, tb[k]);
      DispArgs<R> al = q.al;
      al.tkind = tkind;
      vi.push_back(q.ai);
      vm.push_back(q.am);
      vl.push_back(al);
      vf.push_back(q.af);
      const DispShape *c[4] = {&q.ci, &q.cm, &q.cl, &q.cf};
      DispShape *m[4] = {&p.ci, &p.cm, &p.cl, &p.cf};
      for (int u = 0; u < 4; ++u) {  // one block size and shared-memory size per launch: the largest
        bk[u * n + k + 1] = bk[u * n + k] + c[u]->blocks;
        m[u]->blocks = bk[u * n + k + 1];
        m[u]->threads = std::max(m[u]->threads, c[u]->threads);
        m[u]->smem = std::max(m[u]->smem, c[u]->smem);
      }
    }
    upload(gi, vi);
    upload(gm, vm);
    upload(gl, vl);
    upload(gf, vf);
    upload(blk, bk);
  }

  void run(cudaStream_t s) override {
    const Spectral &sp = *sp0;
    const int nb = uniform ? B : 1, n = B + 1;
    DispGroup<R> g[4];
    const DevBuf *t[4] = {&gi, &gm, &gl, &gf};
    for (int q = 0; q < 4; ++q) g[q] = {t[q]->as<const DispArgs<R>>(), blk.as<const int>() + q * n, B};
    auto grp = [&](int q) { return uniform ? nullptr : &g[q]; };
    disp_ax0_step<R>(sp, p.ai, p.ci, nb, s, grp(0));
    if (dim == 3) disp_mid<R>(sp, true, p.am, p.cm, nb, s, grp(1));
    pixels<R>(sp, tkind, p.al, p.cl, nb, s, grp(2));
    if (dim == 3) disp_mid<R>(sp, false, p.am, p.cm, nb, s, grp(1));
    disp_ax0_dots<R>(sp, p.af, p.cf, nb, s, grp(3));
  }
};

}  // namespace

DispBatch *disp_batch_create(const std::vector<DispProblem> &probs, int tkind, bool uniform, bool fp64) {
  if (fp64) return new DispBatchR<double>(probs, tkind, uniform);
  return new DispBatchR<float>(probs, tkind, uniform);
}
void disp_batch_destroy(DispBatch *b) { delete b; }
void disp_batch_run(DispBatch *b, cudaStream_t s) { b->run(s); }

}  // namespace musg
