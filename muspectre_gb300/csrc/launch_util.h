// Launch helpers shared by the CUDA translation units.
#pragma once

#include <mutex>
#include <set>

#include "musg_internal.h"

namespace musg {

inline int optin_smem() {
  static int v = 0;
  if (v == 0) {
    int dev = 0;
    MUSG_CUDA(cudaGetDevice(&dev));
    int b = 0;
    MUSG_CUDA(cudaDeviceGetAttribute(&b, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    v = b - 2048;  // room for the static shared memory of the reductions
  }
  return v;
}

// raise the dynamic shared-memory limit of a kernel once (keyed by its address)
template <typename K> void allow_smem(K kernel) {
  static std::mutex mu;
  static std::set<const void *> done;
  const void *key = (const void *)kernel;
  std::lock_guard<std::mutex> lock(mu);
  if (done.count(key)) return;
  MUSG_CUDA(cudaFuncSetAttribute(key, cudaFuncAttributeMaxDynamicSharedMemorySize, optin_smem()));
  done.insert(key);
}

template <typename R> const R *xi_table(const Spectral &sp, int d);
template <> inline const double *xi_table<double>(const Spectral &sp, int d) { return (const double *)sp.xi64[d]; }
template <> inline const float *xi_table<float>(const Spectral &sp, int d) { return (const float *)sp.xi32[d]; }

}  // namespace musg
