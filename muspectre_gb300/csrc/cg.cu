// Vector kernels of the Newton level: sums, updates, means, conversions.
// Reductions are deterministic: a fixed block partition, then one block sums the partials
// in a fixed order, so a rerun gives bit-identical scalars.
#include <algorithm>
#include <cstdint>

#include "spectral.cuh"

namespace musg {

constexpr int kRedThreads = 256;
constexpr int kRedMaxBlocks = 2048;

int reduce_blocks(long long n) {
  long long b = (n + kRedThreads * 8 - 1) / (kRedThreads * 8);
  if (b < 1) b = 1;
  if (b > kRedMaxBlocks) b = kRedMaxBlocks;
  return (int)b;
}

// deterministic sum of nparts doubles by one block
__device__ __forceinline__ double sum_partials(const double *partial, int nparts) {
  double v = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) v += partial[i];
  return block_sum(v);
}

// ------------------------------------------------------------------ sums
// (a - b)^2 summed
__global__ void k_diff2(const double *__restrict__ a, const double *__restrict__ b, long long n, double *partial) {
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double d = a[i] - b[i];
    acc += d * d;
  }
  const double bs = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
}

__global__ void k_sum_to(const double *partial, int nparts, double *out) {
  const double v = sum_partials(partial, nparts);
  if (threadIdx.x == 0) *out = v;
}

void diff2_device(const double *a, const double *b, long long n, double *partial, double *out, cudaStream_t s) {
  const int nb = reduce_blocks(n);
  k_diff2<<<nb, kRedThreads, 0, s>>>(a, b, n, partial);
  MUSG_CHECK_LAUNCH();
  k_sum_to<<<1, 1024, 0, s>>>(partial, nb, out);
  MUSG_CHECK_LAUNCH();
}

// F += x; partial sums of x.x and F.F (after the update)
template <typename R>
__global__ void k_newton_update(double *__restrict__ F, const R *__restrict__ x, long long n, double *partial,
                                int nparts) {
  double axx = 0.0, aff = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double xv = (double)x[i];
    const double f = F[i] + xv;
    F[i] = f;
    axx += xv * xv;
    aff += f * f;
  }
  const double s1 = block_sum(axx);
  if (threadIdx.x == 0) partial[blockIdx.x] = s1;
  __syncthreads();
  const double s2 = block_sum(aff);
  if (threadIdx.x == 0) partial[nparts + blockIdx.x] = s2;
}

// line-search trial F = F0 + lam x; partial sums of x.x (the full Newton increment)
// and F.F
template <typename R>
__global__ void k_newton_trial(double *__restrict__ F, const double *__restrict__ F0, const R *__restrict__ x,
                               double lam, long long n, double *partial, int nparts) {
  double axx = 0.0, aff = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double xv = (double)x[i];
    const double f = F0[i] + lam * xv;
    F[i] = f;
    axx += xv * xv;
    aff += f * f;
  }
  const double s1 = block_sum(axx);
  if (threadIdx.x == 0) partial[blockIdx.x] = s1;
  __syncthreads();
  const double s2 = block_sum(aff);
  if (threadIdx.x == 0) partial[nparts + blockIdx.x] = s2;
}

__global__ void k_sum2_to(const double *partial, int nparts, double *out) {
  const double a = sum_partials(partial, nparts);
  __syncthreads();
  const double b = sum_partials(partial + nparts, nparts);
  if (threadIdx.x == 0) {
    out[0] = a;
    out[1] = b;
  }
}

template <typename R>
void newton_update(double *F, const R *x, long long n, double *partial, double *out, cudaStream_t s) {
  const int nb = reduce_blocks(n);
  k_newton_update<R><<<nb, kRedThreads, 0, s>>>(F, x, n, partial, nb);
  MUSG_CHECK_LAUNCH();
  k_sum2_to<<<1, 1024, 0, s>>>(partial, nb, out);
  MUSG_CHECK_LAUNCH();
}

template <typename R>
void newton_trial(double *F, const double *F0, const R *x, double lam, long long n, double *partial, double *out,
                  cudaStream_t s) {
  const int nb = reduce_blocks(n);
  k_newton_trial<R><<<nb, kRedThreads, 0, s>>>(F, F0, x, lam, n, partial, nb);
  MUSG_CHECK_LAUNCH();
  k_sum2_to<<<1, 1024, 0, s>>>(partial, nb, out);
  MUSG_CHECK_LAUNCH();
}

// per-component means of a field [ncomp][npx]: deterministic block sums, then one
// block per component in a fixed order
__global__ void k_plane_sums(const double *__restrict__ f, long long npx, double *partial) {
  const double *fc = f + (long long)blockIdx.y * npx;
  double v = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npx; i += (long long)gridDim.x * blockDim.x)
    v += fc[i];
  const double bs = block_sum(v);
  if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = bs;
}

__global__ void k_plane_finish(const double *partial, int nparts, double scale, double *out) {
  const double v = sum_partials(partial + blockIdx.x * nparts, nparts);
  if (threadIdx.x == 0) out[blockIdx.x] = v * scale;
}

void plane_means(const double *f, int ncomp, long long npx, double *partial, double *out, cudaStream_t s) {
  const int nb = std::min(reduce_blocks(npx), 1024);
  k_plane_sums<<<dim3(nb, ncomp), kRedThreads, 0, s>>>(f, npx, partial);
  MUSG_CHECK_LAUNCH();
  k_plane_finish<<<ncomp, 1024, 0, s>>>(partial, nb, 1.0 / (double)npx, out);
  MUSG_CHECK_LAUNCH();
}

template <typename Rd, typename Rs>
__global__ void k_convert(Rd *__restrict__ dst, const Rs *__restrict__ src, long long n, double scale) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = Rd((double)src[i] * scale);
}

template <typename Rd, typename Rs>
void convert(Rd *dst, const Rs *src, long long n, double scale, cudaStream_t s) {
  k_convert<Rd, Rs><<<reduce_blocks(n), kRedThreads, 0, s>>>(dst, src, n, scale);
  MUSG_CHECK_LAUNCH();
}

template void newton_update<double>(double *, const double *, long long, double *, double *, cudaStream_t);
template void newton_update<float>(double *, const float *, long long, double *, double *, cudaStream_t);
template void newton_trial<double>(double *, const double *, const double *, double, long long, double *, double *,
                                   cudaStream_t);
template void newton_trial<float>(double *, const double *, const float *, double, long long, double *, double *,
                                  cudaStream_t);
template void convert<double, double>(double *, const double *, long long, double, cudaStream_t);
template void convert<float, double>(float *, const double *, long long, double, cudaStream_t);
template void convert<double, float>(double *, const float *, long long, double, cudaStream_t);

}  // namespace musg
