// The displacement-space CG of the mixed method (disp.cuh): launches of its passes.
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
__global__ void k_disp_start(CGState *st, const double *rhs2, const double *range2, double tol, int maxiter) {
  const double in = *range2, all = rhs2 ? *rhs2 : in;
  // FP32 noise of the transform is not a part outside the range
  const double out = all - in;
  st->xscale = sqrt(in);
  st->out2 = out > 1e-5 * all ? out / in : 0.0;
  st->rdr = 1.0 + st->out2;
  st->rhs_norm2 = all / in;
  st->tol2 = tol * tol * (all / in);
  st->alpha = st->beta = st->pAp = 0.0;
  st->iter = 0;
  st->maxiter = maxiter;
  st->ticket = 0;
  // solver_cg.cc:76-77: the first iteration is forced
  st->active = st->go = maxiter > 0 ? 1 : 0;
}

// r = -b / |b|, x = 0.  The points of the plane k_last = 0 come in pairs (k, -k) of one
// real field; rounding leaves b unsymmetric there, the operator's inverse transform
// drops that part and no iteration could reduce it, so each pair takes its mean (in a
// residual accumulated over Newton steps the rounding is that of the largest one, and
// the CG stalled on it).
__global__ void k_disp_init(const float2 *__restrict__ b, float2 *__restrict__ r, float2 *__restrict__ x, int D, int n0,
                            int n1, int nh, const CGState *st) {
  const float c = (float)(-1.0 / st->xscale);
  const unsigned rows = (unsigned)D * n0 * n1, n = rows * (unsigned)nh;  // n1: 1 in 2-D
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float2 v = b[i];
    if (i % nh == 0) {
      const unsigned row = i / nh, k1 = row % n1, dk0 = row / n1, k0 = dk0 % n0;
      const unsigned m0 = k0 ? n0 - k0 : 0, m1 = k1 ? n1 - k1 : 0;
      const float2 w = b[((size_t)(dk0 - k0 + m0) * n1 + m1) * nh];
      v = make_float2(0.5f * (v.x - w.x), 0.5f * (v.y + w.y));  // xi is odd: v(-k) = -conj v(k)
    }
    r[i] = make_float2(c * v.x, c * v.y);
    x[i] = make_float2(0.f, 0.f);
  }
}

// the fourth sums of the blocks, in a fixed order
__global__ void k_disp_sum(const double *partial, int nparts, double *out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += partial[4 * i + 3];
  s = block_sum(s);
  if (threadIdx.x == 0) *out = s;
}

template <typename R> DispProb<R> disp_prob(Spectral &sp, const DispVectors &v, CGState *st, double *partial) {
  using T = typename V2<R>::T;
  sp.ensure32();
  DispProb<R> pb;
  pb.spec = (T *)sp.spec32;
  pb.r = (T *)v.r;
  pb.q = (T *)v.q;
  pb.p = (T *)v.p;
  pb.x = (T *)v.x;
  pb.st = st;
  pb.partial = partial;
  return pb;
}

void pixels(const Spectral &sp, int tkind, const DispArgs<float> &a, const DispShape &c, int B, cudaStream_t s,
            const DispGroup<float> *grp) {
  if (sp.g.dim == 2) disp_pixels<float, 2>(tkind, sp.tp[1], a, c, B, s, grp);
  else disp_pixels<float, 3>(tkind, sp.tp[2], a, c, B, s, grp);
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
void forward_to(Spectral &sp, DispProb<R> pb, int tkind, const double *in, double *prev, double in_scale, bool accumulate,
                double *sum2, cudaStream_t s) {
  DispPasses<R> p = disp_passes<R>(sp, pb);
  p.af.gated = p.am.gated = p.al.gated = 0;
  p.al.in64 = in;
  p.al.in_prev = prev;
  p.al.in_scale = in_scale;
  p.af.accumulate = accumulate ? 1 : 0;
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

void disp_residual(Spectral &sp, void *rhat, const double *field, double *prev, double scale, bool accumulate,
                   double *partial, double *norm2, cudaStream_t s) {
  DispVectors v;
  v.q = rhat;
  forward_to<float>(sp, disp_prob<float>(sp, v, nullptr, partial), TK_PLAIN, field, prev, scale, accumulate, norm2, s);
}

void disp_start(Spectral &sp, const DispVectors &v, const void *rhat, CGState *st, double tol, int maxiter,
                const double *rhs2, const double *range2, cudaStream_t s) {
  const long long n = disp_nk(sp) * sp.g.dim;
  if (n > 0xf0000000ll) throw Error(MUSG_ERR_ARGUMENT, "grid too large for the mixed method");
  k_disp_start<<<1, 1, 0, s>>>(st, rhs2, range2, tol, maxiter);
  MUSG_CHECK_LAUNCH();
  k_disp_init<<<reduce_blocks(n), 256, 0, s>>>((const float2 *)rhat, (float2 *)v.r, (float2 *)v.x, sp.g.dim,
                                                 sp.g.n[0], sp.g.dim == 3 ? sp.g.n[1] : 1, disp_nh(sp), st);
  MUSG_CHECK_LAUNCH();
}

void disp_iteration(Spectral &sp, int tkind, const TangentData<float> &td, const DispVectors &v, CGState *st,
                    double *partial, cudaStream_t s, cudaEvent_t *ev) {
  DispProb<float> pb = disp_prob<float>(sp, v, st, partial);
  pb.td = td;
  const DispPasses<float> p = disp_passes<float>(sp, pb);
  int k = 0;
  auto mark = [&]() {
    if (ev) MUSG_CUDA(cudaEventRecord(ev[k++], s));
  };
  mark();
  disp_ax0_step<float>(sp, p.ai, p.ci, 1, s, nullptr);
  mark();
  if (sp.g.dim == 3) {
    disp_mid<float>(sp, true, p.am, p.cm, 1, s, nullptr);
    mark();
  }
  pixels(sp, tkind, p.al, p.cl, 1, s, nullptr);
  mark();
  if (sp.g.dim == 3) {
    disp_mid<float>(sp, false, p.am, p.cm, 1, s, nullptr);
    mark();
  }
  disp_ax0_dots<float>(sp, p.af, p.cf, 1, s, nullptr);
  mark();
}

void disp_solution(Spectral &sp, const DispVectors &v, CGState *st, float *x, cudaStream_t s) {
  inverse_from<float>(sp, disp_prob<float>(sp, v, st, nullptr), true, x, s);
}

void disp_operator(Spectral &sp, int tkind, const TangentData<float> &td, const double *in, void *qhat, float *out,
                   double *partial, cudaStream_t s) {
  DispVectors v;
  v.q = qhat;
  DispProb<float> pb = disp_prob<float>(sp, v, nullptr, partial);
  pb.td = td;
  forward_to<float>(sp, pb, tkind, in, nullptr, 1.0, false, nullptr, s);
  inverse_from<float>(sp, pb, false, out, s);
}

// ------------------------------------------------------------------ batches
// problems of one grid: a device table indexed by blockIdx.y; of different grids: per
// pass a table of arguments and the prefix sums of the problems' blocks
struct DispBatch {
  bool uniform = true;
  int B = 0, dim = 0, tkind = 0;
  Spectral *sp0 = nullptr;
  DispPasses<float> p;                      // uniform: the shared shapes; else the launches' sizes
  DevBuf tab, gi, gm, gl, gf, blk;          // tables; blk: four prefix sums of B + 1
};

template <typename T> static void upload(DevBuf &d, const std::vector<T> &v) {
  d.alloc(v.size() * sizeof(T));
  MUSG_CUDA(cudaMemcpy(d.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
}

DispBatch *disp_batch_create(const std::vector<DispProblem> &probs, int tkind, bool uniform) {
  auto b = std::make_unique<DispBatch>();
  b->uniform = uniform;
  b->B = (int)probs.size();
  b->sp0 = probs[0].sp;
  b->dim = b->sp0->g.dim;
  b->tkind = tkind;
  std::vector<DispProb<float>> tab;
  for (const DispProblem &q : probs) {
    DispProb<float> pb = disp_prob<float>(*q.sp, q.v, q.st, q.partial);
    pb.td = q.td;
    tab.push_back(pb);
  }
  if (uniform) {
    upload(b->tab, tab);
    b->p = disp_passes<float>(*b->sp0, DispProb<float>{});
    for (DispArgs<float> *a : {&b->p.ai, &b->p.am, &b->p.al, &b->p.af}) a->tab = b->tab.as<DispProb<float>>();
    return b.release();
  }
  const int n = b->B + 1;
  std::vector<DispArgs<float>> gi, gm, gl, gf;
  std::vector<int> blk(4 * n, 0);
  for (int k = 0; k < b->B; ++k) {
    Spectral &sp = *probs[k].sp;
    if (sp.g.dim != b->dim || disp_finite(sp) != disp_finite(*b->sp0))
      throw Error(MUSG_ERR_ARGUMENT, "a grouped operator needs one dimension, projection and component count");
    const DispPasses<float> p = disp_passes<float>(sp, tab[k]);
    DispArgs<float> al = p.al;
    al.tkind = tkind;
    gi.push_back(p.ai);
    gm.push_back(p.am);
    gl.push_back(al);
    gf.push_back(p.af);
    const DispShape *c[4] = {&p.ci, &p.cm, &p.cl, &p.cf};
    DispShape *m[4] = {&b->p.ci, &b->p.cm, &b->p.cl, &b->p.cf};
    for (int q = 0; q < 4; ++q) {  // one block size and shared-memory size per launch: the largest
      blk[q * n + k + 1] = blk[q * n + k] + c[q]->blocks;
      m[q]->blocks = blk[q * n + k + 1];
      m[q]->threads = std::max(m[q]->threads, c[q]->threads);
      m[q]->smem = std::max(m[q]->smem, c[q]->smem);
    }
  }
  upload(b->gi, gi);
  upload(b->gm, gm);
  upload(b->gl, gl);
  upload(b->gf, gf);
  upload(b->blk, blk);
  return b.release();
}

void disp_batch_destroy(DispBatch *b) { delete b; }

void disp_batch_run(DispBatch *b, cudaStream_t s) {
  const Spectral &sp = *b->sp0;
  const int B = b->uniform ? b->B : 1, n = b->B + 1;
  DispGroup<float> g[4];
  const DevBuf *t[4] = {&b->gi, &b->gm, &b->gl, &b->gf};
  for (int q = 0; q < 4; ++q) g[q] = {t[q]->as<const DispArgs<float>>(), b->blk.as<const int>() + q * n, b->B};
  auto grp = [&](int q) { return b->uniform ? nullptr : &g[q]; };
  disp_ax0_step<float>(sp, b->p.ai, b->p.ci, B, s, grp(0));
  if (b->dim == 3) disp_mid<float>(sp, true, b->p.am, b->p.cm, B, s, grp(1));
  pixels(sp, b->tkind, b->p.al, b->p.cl, B, s, grp(2));
  if (b->dim == 3) disp_mid<float>(sp, false, b->p.am, b->p.cm, B, s, grp(1));
  disp_ax0_dots<float>(sp, b->p.af, b->p.cf, B, s, grp(3));
}

}  // namespace musg
