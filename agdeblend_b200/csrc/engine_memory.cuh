// Common helpers of the engine: the FFT tables of the generic kernels, set-up
// timing marks and NVTX ranges (errors and device arrays: device_pool.hpp).
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <memory>
#include <chrono>
#include <functional>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>
#include "agdeblend_gpu.h"
#include "device_pool.hpp"
#include "fast.cuh"
#include "kernels.cuh"
#include "plan.hpp"
#include "wavelet_fast.cuh"
#include "plane_dft.cuh"
#include "time_pair.cuh"
#include "nn_api.hpp"
#include "space_tc.cuh"

namespace agd {

// NVTX range over a scope (host phases of a call, visible in nsys / ncu
// timelines as "agd <phase>")
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// Parts of the engine set-up on stderr when AGD_GPU_TIMING=1: host wall
// clock since the previous mark of this thread, after a device
// synchronisation (reset: start a new sequence without printing).
inline void setup_mark(const char *part, bool reset = false) {
  static const bool on = [] {
    const char *env = std::getenv("AGD_GPU_TIMING");
    return env != nullptr && env[0] == '1';
  }();
  if (!on) return;
  static thread_local std::chrono::steady_clock::time_point t;
  cudaDeviceSynchronize();
  const auto n = std::chrono::steady_clock::now();
  if (!reset)
    std::fprintf(stderr, "agd timing:   set-up/%-12s %8.2f ms\n", part,
                 std::chrono::duration<double, std::milli>(n - t).count());
  t = n;
}

// Distinct FFT lengths with their radix lists and twiddle tables.
template <typename R>
struct FftTable {
  std::vector<FftDesc> descs;
  std::vector<Cx<R>> tw;
  std::map<int, int> index;

  int get(int n) {
    auto it = index.find(n);
    if (it != index.end()) return it->second;
    FftDesc d{};
    d.n = n;
    d.nf = 0;
    int m = n;
    for (int r : {4, 2, 3, 5}) {
      while (m % r == 0) {
        d.radix[d.nf++] = r;
        m /= r;
      }
    }
    for (int p = 7; m > 1; p += 2) {
      while (m % p == 0) {
        if (d.nf >= kMaxFactors) throw DeviceError("FFT length has too many factors");
        d.radix[d.nf++] = p;
        m /= p;
      }
    }
    d.tw_off = (long)tw.size();
    for (int k = 0; k < n; ++k) {
      const double a = -2.0 * 3.14159265358979323846 * (double)k / (double)n;
      Cx<R> w;
      w.x = (R)std::cos(a);
      w.y = (R)std::sin(a);
      tw.push_back(w);
    }
    const int id = (int)descs.size();
    descs.push_back(d);
    index[n] = id;
    return id;
  }
};

static int optin_smem() {
  int dev = 0;
  int v = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return v;
}

}  // namespace agd
