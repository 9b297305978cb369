// Host side of the FFT plans and spectral workspaces.
//
// Twiddles are computed in long double from their definition exp(-2 pi i j/m)
// and rounded once to double and to float; the Bluestein filter DFT_m(conj w)/m is
// formed on the host by a direct DFT with compensated (Kahan) summation.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "launch_util.h"
#include "musg_internal.h"

namespace musg {

std::atomic<unsigned long long> g_launches{0};

void DevBuf::alloc(size_t b) {
  release();
  if (b == 0) return;
  MUSG_CUDA(cudaMalloc(&p, b));
  bytes = b;
}

void DevBuf::release() {
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

namespace {

// radices of a 2/3/5/7-smooth length; returns false when another prime divides n
bool factorize(int n, std::vector<int> &out) {
  out.clear();
  int k = 0;
  while (n % 2 == 0) { n /= 2; ++k; }
  // powers of two: radix 16 as long as possible, the remainder as balanced 8/4
  while (k > 0) {
    if (k >= 4 && k != 5 && k != 6) { out.push_back(16); k -= 4; }
    else if (k == 6) { out.push_back(8); out.push_back(8); k = 0; }
    else if (k == 5) { out.push_back(8); out.push_back(4); k = 0; }
    else if (k == 3) { out.push_back(8); k = 0; }
    else if (k == 2) { out.push_back(4); k = 0; }
    else { out.push_back(2); k = 0; }
  }
  while (n % 9 == 0) { out.push_back(9); n /= 9; }
  for (int r : {3, 5, 7})
    while (n % r == 0) { out.push_back(r); n /= r; }
  return n == 1;
}

int smooth_at_least(int v) {
  for (int m = v;; ++m) {
    int t = m;
    for (int r : {2, 3, 5, 7})
      while (t % r == 0) t /= r;
    if (t == 1) return m;
  }
}

const long double kPi = 3.141592653589793238462643383279502884L;

void *upload(const void *host, size_t bytes) {
  void *d = nullptr;
  MUSG_CUDA(cudaMalloc(&d, bytes));
  MUSG_CUDA(cudaMemcpy(d, host, bytes, cudaMemcpyHostToDevice));
  return d;
}

template <typename T2, typename R>
void *upload_complex(const std::vector<std::complex<long double>> &v) {
  std::vector<T2> h(v.size());
  for (size_t i = 0; i < v.size(); ++i) {
    h[i].x = static_cast<R>(v[i].real());
    h[i].y = static_cast<R>(v[i].imag());
  }
  return upload(h.data(), h.size() * sizeof(T2));
}

// the tables of a length-n transform over m
FftTables fft_tables(int n, int m, int blu) {
  FftTables ft;
  auto &tw = ft.tw, &w = ft.chirp, &bf = ft.bf;
  tw.resize(m);
  for (int j = 0; j < m; ++j) {
    long double a = -2.0L * kPi * (long double)j / (long double)m;
    tw[j] = {cosl(a), sinl(a)};
  }
  if (blu) {
    w.resize(n);
    for (int j = 0; j < n; ++j) {
      long long q = ((long long)j * j) % (2LL * n);
      long double a = -kPi * (long double)q / (long double)n;
      w[j] = {cosl(a), sinl(a)};
    }
    // the filter of b[t] = conj(w[|t|]) on the circle of length m: b is even, so
    // bf[k] = bf[m - k] = (b[0] + 2 sum_{0 < t < n} b[t] cos(2 pi t k / m)) / m, Kahan-compensated
    bf.resize(m);
    std::vector<double> br(n), bi(n), co(m);
    for (int t = 0; t < n; ++t) {
      br[t] = 2.0 * (double)w[t].real();
      bi[t] = -2.0 * (double)w[t].imag();
    }
    for (int j = 0; j < m; ++j) co[j] = (double)tw[j].real();
    for (int k = 0; 2 * k <= m; ++k) {
      double sr = 0.5 * br[0], sc = 0, ir = 0.5 * bi[0], ic = 0;
      int idx = k;
      for (int t = 1; t < n; ++t) {
        const double yr = br[t] * co[idx] - sc, tr = sr + yr;
        sc = (tr - sr) - yr;
        sr = tr;
        const double yi = bi[t] * co[idx] - ic, ti = ir + yi;
        ic = (ti - ir) - yi;
        ir = ti;
        idx += k;
        if (idx >= m) idx -= m;
      }
      bf[k] = bf[(m - k) % m] = {(long double)sr / m, (long double)ir / m};
    }
  }
  return ft;
}

// and on the device, in one precision
template <typename R> void upload_tables(const FftTables &ft, void *&tw, void *&chirp, void *&bf) {
  using T = typename V2<R>::T;
  tw = upload_complex<T, R>(ft.tw);
  if (ft.bf.empty()) return;
  chirp = upload_complex<T, R>(ft.chirp);
  bf = upload_complex<T, R>(ft.bf);
}

}  // namespace

void AxisPlan::factor(int n_) {
  n = n_;
  std::vector<int> rad;
  if (factorize(n, rad)) {
    blu = 0;
    m = n;
  } else {
    blu = 1;
    if (n > (1 << 28)) throw Error(MUSG_ERR_ARGUMENT, "FFT length too large");
    m = smooth_at_least(2 * n - 1);
    factorize(m, rad);
  }
  if ((int)rad.size() > kMaxStages) throw Error(MUSG_ERR_ARGUMENT, "FFT length too large");
  nst = (int)rad.size();
  for (int s = 0; s < nst; ++s) radix[s] = rad[s];
}

void AxisPlan::build(int n_) {
  release();
  factor(n_);
  upload_tables<double>(fft_tables(n, m, blu), tw64, chirp64, bf64);
}

void AxisPlan::release() {
  for (void **p : {&tw64, &chirp64, &bf64}) {
    if (*p) cudaFree(*p);
    *p = nullptr;
  }
}

template <> AxisPlanD<double> AxisPlan::device<double>() const {
  AxisPlanD<double> d{};
  d.n = n; d.m = m; d.nst = nst; d.blu = blu;
  d.rcode = 0;
  for (int s = 0; s < nst; ++s) d.rcode |= (unsigned long long)radix[s] << (5 * s);
  d.tw = (const double2 *)tw64;
  d.chirp = (const double2 *)chirp64;
  d.bf = (const double2 *)bf64;
  return d;
}

namespace {

// arithmetic per point of one radix-r stage, in units of one addition per point: what
// the factor choice below weighs (small composites cost about 2 log2 r and a twiddle,
// the direct primes about r; 24 by measurement: 360 points as 24 x 15 take 6.9 ms of a
// 2-D solve, as 20 x 18 7.1 ms); 0: no such stage
constexpr double kStageCost[33] = {0,  0,  2,  4.5, 4,  8,    6.5, 11, 6.5, 9,  10, 15, 8.5, 18, 13, 12.5, 9,
                                   23, 11, 0,  12,  15, 17,   0,   10, 16,  20, 14, 15, 0,   15, 0,  11};
constexpr bool has_stage(int r) { return r <= 17 || (r <= 32 && r != 19 && r != 23 && r != 29 && r != 31); }
constexpr bool stage_costs_given() {
  for (int r = 2; r <= 32; ++r)
    if ((kStageCost[r] > 0) != has_stage(r)) return false;
  return true;
}
static_assert(stage_costs_given(), "a cost for every radix, and for no other number");
double stage_cost(int r) { return kStageCost[r] + 4.0; }  // + twiddles and a shared-memory round trip

// the cheapest factorisation of m into radices (no heap: the allocation-free projection
// plans with it): two factors up to `widest` (r1 >= r2, possibly 1) if there are any, else
// the fewest up to 17; the number of factors in rad, 0 when a prime above 17 divides m.
// Radices above 17 only where no two up to 17 do, and the most even pair among equals:
// a thread runs a whole butterfly, so on grids that leave the SMs idle the widest one sets
// the time (FP64 32^2 as 8 x 4 instead of one radix 32: 67 -> 32 ms, 64^2 as 8 x 8 instead
// of 32 x 2: 74 -> 43 ms, 64^3 as 8 x 8 instead of 16 x 4: 316 -> 285 ms).
int tile_factor(int m, int widest, int *rad, double &cost) {
  if (widest > 17) {
    const int k = tile_factor(m, 17, rad, cost);
    if (k == 2) return k;
  }
  cost = 1e30;
  int n = 0;
  for (int a = 1; a <= widest; ++a)
    if (m % a == 0 && m / a <= widest) {
      const int b = m / a;
      if (b < a || !has_stage(a) || !has_stage(b)) continue;
      const double c = (a > 1 ? stage_cost(a) : 0.0) + (b > 1 ? stage_cost(b) : 0.0);
      if (c <= cost) {  // a rises: the later of equals is the more even
        cost = c;
        rad[0] = b;
        rad[1] = a;
        n = 2;
      }
    }
  if (n) return n;
  // three or more: peel the factor that leaves the cheapest rest
  for (int a = 17; a >= 2; --a) {
    if (m % a) continue;
    int rest[kMaxStages];
    double c = 0;
    int k = tile_factor(m / a, 17, rest, c);
    if (k == 2 && rest[1] == 1) k = 1;
    if (k == 0 || k + 1 > kMaxStages || c + stage_cost(a) + 1.0 >= cost) continue;
    cost = c + stage_cost(a) + 1.0;
    rad[0] = a;
    for (int q = 0; q < k; ++q) rad[q + 1] = rest[q];
    n = k + 1;
  }
  return n;
}

}  // namespace

void TilePlan::factor(int n_, int widest, int wide_blu, long points, bool smallest) {
  n = n_;
  m = nst = r1 = r2 = blu = 0;
  if (n > (1 << 16)) return;  // longer than any tile: the passes refuse it (m = 0)
  double cost = 0;
  if ((nst = tile_factor(n, widest, radix, cost))) {
    m = n;
  } else {
    // Bluestein: the cheapest m in [2n-1, 2.5n]; the two middle stages share a pass
    blu = 1;
    // the cheapest may be too long for its pass where a shorter one fits (899 in 2-D: 2048
    // points of four components in two buffers are 262 KB, 1800 fit); where none fits, the
    // pass refuses the length
    double best = 1e30;
    for (long most : {points, (long)(1 << 28)}) {
      for (int k = 2 * n - 1; k <= 2 * n - 1 + n / 2 + 16; ++k) {
        int rad[kMaxStages];
        double c = 0;
        const int ns = tile_factor(k, wide_blu, rad, c);
        if (!ns || (ns > 2 && k > most)) continue;
        if (smallest && m) break;
        c *= k;
        if (c < best) {
          best = c;
          m = k;
          nst = ns;
          for (int q = 0; q < ns; ++q) radix[q] = rad[q];
        }
      }
      if (m) break;
    }
    if (!m) throw Error(MUSG_ERR_ARGUMENT, "FFT length too large");
  }
  r1 = nst == 2 ? radix[0] : 0;
  r2 = nst == 2 ? radix[1] : 0;
}

template <typename R> void TilePlan::build(int n_, int dim, long points, const TilePlan *other) {
  release();
  factor(n_, dim == 2 ? 32 : 17, wide_bluestein<R>(n_, dim), points);
  if (!m) return;
  host = other && other->host && other->m == m ? other->host : std::make_shared<const FftTables>(fft_tables(n, m, blu));
  upload_tables<R>(*host, tw, chirp, bf);
}

void TilePlan::release() {
  for (void **p : {&tw, &chirp, &bf}) {
    if (*p) cudaFree(*p);
    *p = nullptr;
  }
  host.reset();
}

template <typename R> TilePlanD<R> TilePlan::device() const {
  using T = typename V2<R>::T;
  TilePlanD<R> d{};
  d.n = n; d.m = m; d.r1 = r1; d.r2 = r2; d.blu = blu; d.nst = nst;
  for (int s = 0; s < nst; ++s) d.rcode |= (unsigned long long)radix[s] << (5 * s);
  d.tw = (const T *)tw;
  d.chirp = (const T *)chirp;
  d.bf = (const T *)bf;
  return d;
}
template TilePlanD<double> TilePlan::device<double>() const;
template TilePlanD<float> TilePlan::device<float>() const;

// fftfreq(n)[k]/L (src/fft/fft_utils.cc:41-56)
static double fft_freq(int n, int k) {
  int N = (n - 1) / 2 + 1;
  return k < N ? (double)k : (double)(-(n / 2) + k - N);
}

void Spectral::init(int dim, const int *res, int ncomp_, int proj_kind_, const double *lengths_,
                    bool allow_even_, bool want32_) {
  release();
  if (dim != 2 && dim != 3) throw Error(MUSG_ERR_ARGUMENT, "only 2- and 3-dimensional grids are supported");
  g.dim = dim;
  g.npx = 1;
  for (int d = 0; d < 3; ++d) g.n[d] = 1;
  for (int d = 0; d < dim; ++d) {
    if (res[d] < 1) throw Error(MUSG_ERR_ARGUMENT, "resolutions must be positive");
    g.n[d] = res[d];
    g.npx *= res[d];
    lengths[d] = lengths_ ? lengths_[d] : 1.0;
  }
  g.nh = g.n[dim - 1] / 2 + 1;
  g.nrows = g.npx / g.n[dim - 1];
  g.nk = g.nrows * g.nh;
  ncomp = ncomp_;
  proj_kind = proj_kind_;
  allow_even = allow_even_;
  want32 = want32_;
  // the tables are the FFT engine's; cells and projections have those of their passes
  // (ensure_tiles)
  for (int d = 0; d < dim; ++d) proj_kind < 0 ? ax[d].build(g.n[d]) : ax[d].factor(g.n[d]);
  // xi tables over the hermitian index range of each axis
  for (int d = 0; d < dim; ++d) {
    int len = (d == dim - 1) ? g.nh : g.n[d];
    std::vector<double> h(len);
    std::vector<float> hf(len);
    for (int k = 0; k < len; ++k) {
      h[k] = fft_freq(g.n[d], k) / lengths[d];
      hf[k] = (float)h[k];
    }
    xi64[d] = upload(h.data(), len * sizeof(double));
    xi32[d] = upload(hf.data(), len * sizeof(float));
  }
  MUSG_CUDA(cudaMalloc(&spec64, (size_t)ncomp * g.nk * sizeof(double2)));
  if (want32) ensure32();
}

template <typename R> long Spectral::tile_points(int axis, long bytes) const {
  const int D = g.dim, sym = D * (D + 1) / 2;
  const bool fin = proj_kind != MUSG_PROJ_SMALL_STRAIN;
  // a pass over a middle axis falls back to one component at a time
  const int pencils = axis == D - 1 ? (fin ? D * D : sym) : axis == 0 ? (fin ? 2 : sym) : 1;
  return bytes / (pencils * 2 * (long)(2 * sizeof(R)));
}
template long Spectral::tile_points<double>(int, long) const;
template long Spectral::tile_points<float>(int, long) const;

void Spectral::ensure_tiles() {
  for (int d = 0; d < g.dim; ++d)
    if (tp64[d].n != g.n[d]) tp64[d].build<double>(g.n[d], g.dim, tile_points<double>(d, optin_smem()), nullptr);
}

void Spectral::ensure32() {
  want32 = true;
  ensure_tiles();
  for (int d = 0; d < g.dim; ++d)
    if (tp32[d].n != g.n[d]) tp32[d].build<float>(g.n[d], g.dim, tile_points<float>(d, optin_smem()), &tp64[d]);
  if (!spec32) MUSG_CUDA(cudaMalloc(&spec32, (size_t)ncomp * g.nk * sizeof(float2)));
}

void Spectral::release() {
  for (auto &a : ax) a.release();
  for (auto &a : tp64) a.release();
  for (auto &a : tp32) a.release();
  for (int d = 0; d < 3; ++d) {
    if (xi64[d]) cudaFree(xi64[d]);
    if (xi32[d]) cudaFree(xi32[d]);
    xi64[d] = xi32[d] = nullptr;
  }
  if (spec64) cudaFree(spec64);
  if (spec32) cudaFree(spec32);
  spec64 = spec32 = nullptr;
}

}  // namespace musg
