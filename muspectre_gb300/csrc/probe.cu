// FP64 FMA throughput probe (instrumentation; no counterpart in the reference).
//
// The FP64 plain method and the FP64 Newton level of the mixed path run FFT and
// pixel-local passes whose arithmetic intensity (about 1 flop per byte) puts them on
// the FP64 FMA pipe rather than on HBM bandwidth on this GPU.  Their roofline needs a
// measured FP64 peak: this kernel keeps every SM's FP64 pipe busy with independent
// fused multiply-add chains (eight per thread, so that the pipe's latency is covered
// by the chains of one warp and the warps of a block) and reports FLOP/s = 2 x FMAs /
// CUDA-event time.
//
// Also the self-test of a bounded wait on an mbarrier (musg_selftest_wait_timeout): a
// wait that nothing completes gives up after a wall-clock limit, records the fault in a
// device word and leaves the device usable.
#include <cstdint>

#include "musg_internal.h"

namespace musg {
namespace {

constexpr int kChains = 8;

__global__ void k_fp64_fma(double *sink, int iters, double a, double b) {
  double v[kChains];
#pragma unroll
  for (int c = 0; c < kChains; ++c) v[c] = (double)(threadIdx.x + c) * 1e-3;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int c = 0; c < kChains; ++c) v[c] = fma(v[c], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < kChains; ++c) s += v[c];
  if (s == 12345.678) sink[0] = s;  // keeps the chains live; never true for these inputs
}

__device__ unsigned int g_wait_fault;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// poll until the phase of the given parity completed or the wall-clock limit ran out
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (unsigned i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && global_ns() - t0 > limit_ns) return false;
  }
}

// Self-test of the bounded wait: one thread waits on an mbarrier that nothing arrives
// at, gives up after limit_ns, records the fault word, and
// the kernel exits (no copy is in flight).
__global__ void k_wait_probe(unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait_bounded(&bar, 0, limit_ns)) atomicOr(&g_wait_fault, 1u);
}

}  // namespace

void wait_probe(unsigned long long limit_ns, cudaStream_t s) {
  k_wait_probe<<<1, 32, 0, s>>>(limit_ns);
  MUSG_CHECK_LAUNCH();
}

unsigned *wait_fault_word() {
  static unsigned *p = [] {
    void *q = nullptr;
    MUSG_CUDA(cudaGetSymbolAddress(&q, g_wait_fault));
    return static_cast<unsigned *>(q);
  }();
  return p;
}

double fp64_fma_tflops(cudaStream_t s) {
  int dev = 0, nsm = 0;
  MUSG_CUDA(cudaGetDevice(&dev));
  MUSG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  double *sink = nullptr;
  MUSG_CUDA(cudaMalloc(&sink, sizeof(double)));
  cudaEvent_t e0, e1;
  MUSG_CUDA(cudaEventCreate(&e0));
  MUSG_CUDA(cudaEventCreate(&e1));
  const int threads = 256, blocks = nsm * 8, iters = 4096;
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    MUSG_CUDA(cudaEventRecord(e0, s));
    k_fp64_fma<<<blocks, threads, 0, s>>>(sink, iters, 0.999999, 1e-9);
    MUSG_CHECK_LAUNCH();
    MUSG_CUDA(cudaEventRecord(e1, s));
    MUSG_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    MUSG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (rep > 0 && ms < best) best = ms;  // the first launch warms up
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  const double flops = 2.0 * kChains * (double)iters * threads * (double)blocks;
  return flops / (best * 1e-3) / 1e12;
}

}  // namespace musg
