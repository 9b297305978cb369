// Internal declarations shared by the CUDA translation units and the host API of
// libmusg.  Nothing here is part of the C ABI (include/musg.h is).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <complex>
#include <cstdint>
#include <functional>
#include <memory>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/musg.h"

namespace musg {

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};


// Runs f, maps an exception to a status code and the calling thread's last-error
// message (the C-ABI convention of every musg_* entry point)
int guarded(const std::function<void()> &f);

#define MUSG_CUDA(call)                                                              \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess)                                                           \
      throw ::musg::Error(e_ == cudaErrorMemoryAllocation ? MUSG_ERR_MEMORY          \
                                                          : MUSG_ERR_CUDA,           \
                          std::string(#call) + ": " + cudaGetErrorString(e_));       \
  } while (0)

// kernels launched by the library in this process (graph replays add their nodes)
extern std::atomic<unsigned long long> g_launches;

#define MUSG_CHECK_LAUNCH()                 \
  do {                                      \
    ::musg::g_launches.fetch_add(1);        \
    MUSG_CUDA(cudaGetLastError());          \
  } while (0)

// Programmatic dependent launch: a kernel launched with launch_pdl may be scheduled
// while the previous kernel of its stream finishes (its launch overlaps that tail);
// it calls dep_wait() before it reads anything another kernel writes, which returns once
// the previous grid has completed and its memory is visible.  No kernel here triggers
// early, so the previous grid's blocks have all exited before any block of the next one
// runs.  (Triggering at the start, so that the next kernel's blocks are placed while the
// last ones of a grid run, packed them on the SMs that were free first: 35^3 FP64 solves
// 75 -> 97 ms, FP32 ones unchanged.)
#ifdef __CUDACC__
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... KArgs, typename... Args>
void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  MUSG_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}
#endif

template <typename R> struct V2;
template <> struct V2<float> { using T = float2; };
template <> struct V2<double> { using T = double2; };

constexpr int kMaxStages = 12;  // 5 bits per stage in AxisPlanD::rcode
constexpr int kMaxMaterials = 256;
// MaterialHyperElastoPlastic1 mode (MatParams::logm_mode) with the consistent tangent
constexpr int kHep1Consistent = 2;

// ---------------------------------------------------------------- FFT plans
// Device view of a 1-D FFT plan for one axis.  A length-n transform runs as a
// Stockham mixed-radix FFT of length m (m == n), or, when n has a prime factor
// above 7, as Bluestein's chirp-z algorithm over a 2/3/5/7-smooth m >= 2n-1.
template <typename R> struct AxisPlanD {
  int n;
  int m;
  int nst;
  int blu;
  unsigned long long rcode;  // radix of stage s in bits [5s, 5s+5)
  const typename V2<R>::T *tw;    // m entries: exp(-2 pi i j / m)
  const typename V2<R>::T *chirp; // n entries: exp(-pi i j^2 / n)     (Bluestein)
  const typename V2<R>::T *bf;    // m entries: DFT_m(conj chirp)/m     (Bluestein)
};

struct AxisPlan {
  int n = 0, m = 0, nst = 0, blu = 0;
  int radix[kMaxStages] = {0};
  void *tw64 = nullptr, *chirp64 = nullptr, *bf64 = nullptr;  // device tables
  void factor(int n);  // host only; build() also makes the tables
  void build(int n);
  void release();
  template <typename R> AxisPlanD<R> device() const;
};

// Plan of the in-place tile transforms (tile_fft.cuh): m = r1 r2 in two stages (r1 = 0:
// three or more factors, the radix of stage s in bits [5s, 5s+5) of rcode), blu: a
// Bluestein transform of length n over m.
template <typename R> struct TilePlanD {
  int n, m, r1, r2, blu, nst;
  unsigned long long rcode;
  const typename V2<R>::T *tw;     // m entries: exp(-2 pi i j / m)
  const typename V2<R>::T *chirp;  // n entries (Bluestein)
  const typename V2<R>::T *bf;     // m entries (Bluestein)
};
struct FftTables {  // on the host: twiddles W_m^j; Bluestein: the chirp and the filter
  std::vector<std::complex<long double>> tw, chirp, bf;
};
struct TilePlan {
  int n = 0, m = 0, r1 = 0, r2 = 0, blu = 0, nst = 0;
  int radix[kMaxStages] = {0};
  void *tw = nullptr, *chirp = nullptr, *bf = nullptr;  // device tables of one precision
  std::shared_ptr<const FftTables> host;                // what they were rounded from
  // factors only (host), two up to `widest` (17, or 32 for the axes of a 2-D grid; those of a
  // Bluestein length up to `wide_blu`); build() also makes the device tables, from those of
  // the other precision's plan where both have one length.  points: the
  // longest plan of three or more factors that fits the axis' passes; smallest: the shortest
  // Bluestein length instead of the cheapest
  void factor(int n, int widest, int wide_blu, long points, bool smallest = false);
  template <typename R> void build(int n, int dim, long points, const TilePlan *other);
  void release();
  template <typename R> TilePlanD<R> device() const;
  int buffers() const { return r1 ? 1 : 2; }  // tile buffers a transform needs
};
// The largest radix of a Bluestein length on an axis of n points.  On 2-D grids two wide
// radices replace three factors: in FP32 at every length (139^2 12.3 -> 8.9 ms, 701 x 211
// 16.5 -> 14.5), in FP64, where they spill, only above 256 points (157 x 149 109 -> 161 ms
// with them)
template <typename R> int wide_bluestein(int n, int dim) { return dim == 2 && (sizeof(R) == 4 || n > 256) ? 32 : 17; }

// ---------------------------------------------------------------- geometry
struct Geom {
  int dim = 0;
  int n[3] = {1, 1, 1};     // real grid, row-major, n[dim-1] is the last axis
  int nh = 0;               // n_last/2 + 1
  long long npx = 0;        // pixels
  long long nk = 0;         // hermitian k-points
  long long nrows = 0;      // npx / n_last
  int nlast() const { return n[dim - 1]; }
};

// Per-pixel tangent representation used by the CG operator (pass A prologue).
enum TangentKind : int {
  TK_PLAIN = 0,   // no tangent: input field copied (FFT engine / projection)
  TK_SMALL = 1,   // small strain, isotropic: dP = lam tr(dF) I + mu (dF + dF^T)
  TK_FINITE = 2,  // finite strain, isotropic PK2/GL: dP = dF S + F (lam tr(A) I + mu (A + A^T)), A = F^T dF
  TK_KPRIME = 3,  // j-independent Kirchhoff tangent: dP(i,m) = sum_n K'(i,m,n) sum_j dF(j,n)
  TK_MIXED = 4,   // per-pixel choice between TK_FINITE and TK_KPRIME by material law
  TK_FISO = 5,    // TK_FINITE with S rebuilt from F per application (isotropic LE1/LE3/LE4)
  TK_GSMALL = 6,  // small strain, per-material stiffness C (MaterialLinearElasticGeneric): dP = C:de
  TK_GFINITE = 7, // finite strain, per-material C: dP = dF S + F (C:(F^T dF))
  TK_ANYFIN = 9,  // the displacement-space pixel pass (disp.cuh): any finite-strain kind, by DispArgs::tkind
  TK_FULL = 8,    // stored per-pixel tangent K(i,m,j,n) (D^4 planes): dP = K:dF (the consistent
                  // elasto-plastic tangent, and the elastic pixels of a cell that has it)
};

// A caller's stop flag (a host int another thread may set): nonzero ends a running
// solve at its next check with MUSG_ERR_RUNTIME "cancelled while running".
inline void check_stop(const int *flag) {
  if (flag && __atomic_load_n(flag, __ATOMIC_RELAXED) != 0) throw Error(MUSG_ERR_RUNTIME, "cancelled while running");
}

// Device data the CG operator reads (precision R).
template <typename R> struct TangentData {
  const R *lam = nullptr;   // [npx]
  const R *mu = nullptr;    // [npx]
  const R *F = nullptr;     // [D*D][npx]  (finite strain): F in FP64, F - I in FP32
  const R *S = nullptr;     // [D*D][npx] PK2 stress (finite strain, isotropic)
  const R *Kp = nullptr;    // [D^3][npx]  (Kirchhoff tangent)
  const uint8_t *mat = nullptr;      // [npx] material index (TK_MIXED, C)
  const uint8_t *law_kind = nullptr; // [kMaxMaterials]: TK_FINITE or TK_KPRIME (TK_MIXED)
  const R *C = nullptr;     // [nmat][D^4] stiffness per material (TK_GSMALL / TK_GFINITE)
  const R *Kt = nullptr;    // [D^4][npx] per-pixel tangent planes, entry (i + D m) + D^2 (j + D n) (TK_FULL)
};

// CG scalar state, resident on the device (all FP64).
struct CGState {
  double rdr;        // r.r of the current residual
  double rhs_norm2;  // rhs.rhs
  double tol2;       // tol^2 * rhs.rhs
  double alpha, beta, pAp;
  int iter;          // iterations of this solve
  int maxiter;
  int active;        // 1 while the loop runs
  int ticket;        // blocks of the running kernel that have written their partial sum
  unsigned long long counter;  // cumulative iterations (SolverBase::counter)
  // displacement-space iteration (disp.cuh): whether another operator application follows
  // (active: the update pass is still due), and the part of |rhs|^2 outside the range of
  // the projection
  int go;
  double out2;
  double xscale;  // the norm of the right-hand side, by which that solve is scaled
};

// ---------------------------------------------------------------- spectral ops
// Workspace + plans for one grid; one instance per cell / FFT engine / projection.
struct Spectral {
  Geom g;
  int ncomp = 0;            // components per pixel
  int proj_kind = -1;       // MUSG_PROJ_* (-1: none)
  bool allow_even = false;
  double lengths[3] = {1, 1, 1};
  AxisPlan ax[3];
  TilePlan tp64[3], tp32[3];  // the same axes for the displacement-space passes (disp.cu), by ensure_tiles, ensure32
  template <typename R> const TilePlan &tile(int axis) const { return sizeof(R) == 8 ? tp64[axis] : tp32[axis]; }
  // per-axis xi_d(k) = fftfreq_d(k)/L_d over the hermitian index range, FP64 and FP32
  void *xi64[3] = {nullptr, nullptr, nullptr};
  void *xi32[3] = {nullptr, nullptr, nullptr};
  void *spec64 = nullptr;   // [ncomp][nk] complex double
  void *spec32 = nullptr;   // [ncomp][nk] complex float
  bool want32 = false;
  void init(int dim, const int *res, int ncomp, int proj_kind, const double *lengths,
            bool allow_even, bool want32);
  // points of a pencil of two buffers in `bytes` of shared memory, for the pass over `axis`
  // that holds the most pencils at once (disp_launch.cuh)
  template <typename R> long tile_points(int axis, long bytes) const;
  void ensure_tiles();
  void ensure32();
  void release();
};

// Device word set by a kernel whose bounded wait ran out (probe.cu); its device address,
// for a stream-ordered read by the host
unsigned *wait_fault_word();
// one block that waits on an mbarrier nothing arrives at, bounded by limit_ns
// (self-test of the bounded waits: it sets the fault word and exits)
void wait_probe(unsigned long long limit_ns, cudaStream_t s);

// The FFT engine's passes (last axis, middle axis, first axis): the most threads per block,
// threads per block, and the shared memory a block aims for
constexpr int kPassThreads = 512;
constexpr int kEngineThreads[3] = {256, 256, 256};
constexpr long kEngineBytes[3] = {73728, 49152, 73728};

// Pass launchers (spectral_*.cu).  All run on `stream`.
//  fwd: real field [ncomp][npx] (scaled) -> spectrum (r2c over all axes)
//  inv: spectrum -> real field (c2r, unnormalised, scaled)
template <typename R>
void spectral_forward(Spectral &sp, const R *in, R scale, cudaStream_t s);
template <typename R>
void spectral_inverse(Spectral &sp, R *out, R scale, cudaStream_t s);

// ---------------------------------------------------------------- displacement-space CG (disp.cu)
// The CG solver and the projection (disp.cuh), in FP64 and, for the mixed method's inner
// solve, in FP32 (R).  A vector in the range of the projection is D complex values per
// half-spectrum point, [D][disp_nk].
struct DispVectors {
  void *r = nullptr, *q = nullptr, *p = nullptr, *x = nullptr;
};
// stored k-points of the last axis (the Nyquist column of an even axis is zero), and of
// the half spectrum
inline int disp_nh(const Spectral &sp) { return (sp.g.nlast() + 1) / 2; }
inline long long disp_nk(const Spectral &sp) { return sp.g.nrows * disp_nh(sp); }
template <typename R> size_t disp_vector_bytes(const Spectral &sp) {
  return (size_t)disp_nk(sp) * sp.g.dim * 2 * sizeof(R);
}
// rhat = the projection of scale * field (FP64 planes), through the tangent unless tkind is
// TK_PLAIN; or with prev of prev - field, after which prev = field.  *norm2 (may be null) =
// |rhat|^2, a device double
template <typename R>
void disp_residual(Spectral &sp, int tkind, const TangentData<R> &td, void *rhat, const double *field, double *prev,
                   double scale, double *partial, double *norm2, cudaStream_t s);
// r64 += r32 (an FP32 rhat), then r32 = r64 rounded, *norm2 = |r64|^2 summed in FP64
void disp_accumulate(Spectral &sp, void *r64, void *r32, double *partial, double *norm2, cudaStream_t s);
// state and vectors of a solve A x = rhs for the rhat of its right-hand side, *range2 =
// |rhat|^2; *out2 (null: 0) is the part of |rhs|^2 outside the range of the projection,
// which stays in the residual (device doubles)
template <typename R>
void disp_start(Spectral &sp, const DispVectors &v, const void *rhat, CGState *st, double tol, int maxiter,
                const double *out2, const double *range2, cudaStream_t s);
// one CG iteration: five passes (3-D) or three (2-D)
template <typename R>
void disp_iteration(Spectral &sp, int tkind, const TangentData<R> &td, const DispVectors &v, CGState *st,
                    double *partial, cudaStream_t s, cudaEvent_t *ev = nullptr);
// the solution of the state's solve as real component planes
template <typename R>
void disp_solution(Spectral &sp, const DispVectors &v, CGState *st, R *x, cudaStream_t s);
// the real field of a vector
template <typename R> void disp_field(Spectral &sp, void *qhat, R *out, cudaStream_t s);
// out = G(K:in) of a real field (FP64 planes in), without the tangent when tkind is
// TK_PLAIN; in and out may be the same
template <typename R>
void disp_operator(Spectral &sp, int tkind, const TangentData<R> &td, const double *in, R *out, cudaStream_t s);
// an FP64 vector in FP32
void disp_convert(const Spectral &sp, const void *v64, void *v32, cudaStream_t s);
// iterations of several problems per launch: of one grid (the solo kernels, problem =
// blockIdx.y), or of different grids (each owning a range of the blocks)
struct DispProblem {
  Spectral *sp;
  DispVectors v;
  CGState *st;
  double *partial;
  TangentData<float> td32;
  TangentData<double> td64;
};
struct DispBatch;
DispBatch *disp_batch_create(const std::vector<DispProblem> &probs, int tkind, bool uniform, bool fp64);
void disp_batch_destroy(DispBatch *b);
void disp_batch_run(DispBatch *b, cudaStream_t s);

// ---------------------------------------------------------------- CG kernels (cg.cu)
int reduce_blocks(long long n);
// per-component means of a field [ncomp][npx] into out[ncomp] (device); partial
// holds ncomp * 1024 doubles
void plane_means(const double *f, int ncomp, long long npx, double *partial, double *out, cudaStream_t s);
// sum of (a - b)^2 over n entries into *out (device)
void diff2_device(const double *a, const double *b, long long n, double *partial, double *out, cudaStream_t s);
// y += x (promoting), with the dots x.x and y.y (after the update) into out[0], out[1]
template <typename R>
void newton_update(double *F, const R *x, long long n, double *partial, double *out,
                   cudaStream_t s);
// line-search trial F = F0 + lam x, with x.x and F.F into out[0], out[1]
template <typename R>
void newton_trial(double *F, const double *F0, const R *x, double lam, long long n, double *partial, double *out,
                  cudaStream_t s);
template <typename Rd, typename Rs>
void convert(Rd *dst, const Rs *src, long long n, double scale, cudaStream_t s);

// ---------------------------------------------------------------- materials (materials.cu)
struct MatParams {
  int law;
  int logm_mode;            // HEP1: 0 projector sum (reference), 1 spectral, 2 spectral with the
                            // consistent Kirchhoff->PK1 tangent (kHep1Consistent)
  double lam, mu, K, tau_y0, H;
};

struct MaterialArgs {
  int dim, form;
  long long npx;
  const double *F;          // [D*D][npx]
  double *P;                // [D*D][npx]
  const uint8_t *mat;       // [npx]
  const MatParams *params;  // [nmat]
  const double *lam, *mu;   // [npx] (elastic laws)
  const double *eig;        // [D*D][npx] eigenstrain (LE2), may be null
  const double *Ctab;       // [nmat][D^4] stiffness of MaterialLinearElasticGeneric materials
  // HEP1 state, two buffers each; cur selects the current one
  double *Fprev[2], *be[2], *eps[2];
  int cur;
  // tangent outputs in CG precision (float or double, one of them set)
  double *S64, *Kp64, *Fc64;
  float *S32, *Kp32, *Fc32;
  double *Kfull;            // optional full tangent, AoS [npx][D^4] (API)
  double *Kt64;             // TK_FULL: tangent planes [D^4][npx] in the CG precision (one set)
  float *Kt32;
  int *nonfinite;           // device flag set when a non-finite stress appears
  int has_hep;              // any MaterialHyperElastoPlastic1 pixel in the cell
};
void material_evaluate(const MaterialArgs &a, cudaStream_t s);
void add_macro(double *F, const double *delta_dev, int ncomp, long long npx, cudaStream_t s);
void fill_uniform(double *F, const double *value_dev, int ncomp, long long npx, cudaStream_t s);
// per-pixel Lame planes from the material index and the per-material parameters
void fill_lame(const uint8_t *mat, const MatParams *params, double *lam, double *mu, long long npx, cudaStream_t s);

// AoS (host layout, pixel-major) <-> SoA (component planes) on the device
void aos_to_soa(const double *aos, double *soa, int ncomp, long long npx, cudaStream_t s);
void soa_to_aos(const double *soa, double *aos, int ncomp, long long npx, cudaStream_t s);
void soa_to_aos_complex(const double2 *soa, double2 *aos, int ncomp, long long nk, cudaStream_t s);
void aos_to_soa_complex(const double2 *aos, double2 *soa, int ncomp, long long nk, cudaStream_t s);

// measured FP64 FMA throughput of the current device, TFLOP/s (probe.cu)
double fp64_fma_tflops(cudaStream_t s);

// allocation-free projection on caller device buffers (noalloc.cu)
void noalloc_project(int dim, const int *resolutions, const double *lengths, int kind, int flags,
                     const double *in_device, double *out_device, cudaStream_t s);

// simple device buffer
struct DevBuf {
  void *p = nullptr;
  size_t bytes = 0;
  void alloc(size_t b);
  void release();
  template <typename T> T *as() const { return reinterpret_cast<T *>(p); }
  ~DevBuf() { release(); }
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
};

}  // namespace musg
