// Device memory of the engine: errors, the cache of device blocks
// (DevicePool) and typed device arrays (DevArray).  Host code only.
#pragma once

#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <map>
#include <mutex>
#include <stdexcept>
#include <vector>
#include "plan.hpp"

namespace agd {

struct DeviceError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

static void check(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    char buf[512];
    std::snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    throw DeviceError(buf);
  }
}
#define CK(x) check((x), #x)

// Device blocks of finished problems kept for the next problem on the same
// device: a deblending call allocates its arrays once per call, a fresh
// cudaMalloc of gigabytes costs page mapping that can exceed the solve
// itself, and the fifty small tables of a 40-trace gather cost 0.3 ms of a
// 1.1 ms call in cudaMalloc and cudaFree.  Blocks enter the cache only when
// their engine has waited for the work that used them, so no kernel can
// still use them; a block that an exception releases is freed instead.  A block belongs to the device it was
// allocated on, whichever device is current when it comes back.  Sizes are
// rounded up to kGrain; a request takes the smallest block that fits if that
// is at most twice as large (from kLarge on, twice and kSlack more), so that
// tables leave the blocks of large arrays alone.  At most half the device
// memory is held (AGD_GPU_CACHE=0 disables the cache; agd_gpu_release_cache
// frees it).
class DevicePool {
 public:
  static constexpr size_t kGrain = 512;
  static constexpr size_t kLarge = size_t(1) << 16;
  static constexpr size_t kSlack = size_t(1) << 20;

  static void *take(size_t bytes) {
    bytes = (bytes + kGrain - 1) / kGrain * kGrain;
    if (injected_alloc_failure()) throw DeviceError("injected device allocation failure");
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (enabled()) {
      std::lock_guard<std::mutex> g(mu());
      auto &m = free_blocks()[dev];
      auto it = m.lower_bound(bytes);
      if (it != m.end() && it->first <= 2 * bytes + (bytes >= kLarge ? kSlack : 0)) {
        void *p = it->second;
        held() -= it->first;
        m.erase(it);
        return p;
      }
    }
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      release_device(dev);
      e = cudaMalloc(&p, bytes);
    }
    CK(e);
    std::lock_guard<std::mutex> g(mu());
    blocks()[p] = Block{bytes, dev};
    return p;
  }

  static void put(void *p) {
    if (p == nullptr) return;
    std::lock_guard<std::mutex> g(mu());
    const Block b = blocks()[p];
    // released by an exception: launches before it may still use the block,
    // and cudaFree waits for the device
    if (std::uncaught_exceptions() > 0 || !enabled() ||
        held() + b.bytes > half_memory(b.dev)) {
      blocks().erase(p);
      cudaFree(p);
      return;
    }
    free_blocks()[b.dev].emplace(b.bytes, p);
    held() += b.bytes;
  }

  static void release_device(int dev) {
    std::lock_guard<std::mutex> g(mu());
    auto &m = free_blocks()[dev];
    for (auto &kv : m) {
      held() -= kv.first;
      blocks().erase(kv.second);
      cudaFree(kv.second);
    }
    m.clear();
  }

  static void release_all() {
    std::vector<int> devs;
    {
      std::lock_guard<std::mutex> g(mu());
      for (auto &kv : free_blocks()) devs.push_back(kv.first);
    }
    int cur = 0;
    cudaGetDevice(&cur);
    for (int d : devs) {
      cudaSetDevice(d);
      release_device(d);
    }
    cudaSetDevice(cur);
  }

 private:
  struct Block {
    size_t bytes;
    int dev;
  };
  // half the device's memory, queried once (a memory-information query on
  // every return would cost a driver call each); with the mutex held
  static size_t half_memory(int dev) {
    static std::map<int, size_t> half;
    auto it = half.find(dev);
    if (it != half.end()) return it->second;
    int cur = 0;
    size_t freeb = 0, total = 0;
    cudaGetDevice(&cur);
    if (cur != dev) cudaSetDevice(dev);
    const cudaError_t e = cudaMemGetInfo(&freeb, &total);
    if (cur != dev) cudaSetDevice(cur);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return half[dev] = total / 2;
  }
  static bool enabled() {
    static const bool on = [] {
      const char *env = std::getenv("AGD_GPU_CACHE");
      return !(env != nullptr && env[0] == '0');
    }();
    return on;
  }
  static std::mutex &mu() {
    static std::mutex m;
    return m;
  }
  static std::map<int, std::multimap<size_t, void *>> &free_blocks() {
    static std::map<int, std::multimap<size_t, void *>> m;
    return m;
  }
  static std::map<void *, Block> &blocks() {
    static std::map<void *, Block> m;
    return m;
  }
  static size_t &held() {
    static size_t h = 0;
    return h;
  }
};

template <typename T>
class DevArray {
 public:
  DevArray() = default;
  DevArray(const DevArray &) = delete;
  DevArray &operator=(const DevArray &) = delete;
  DevArray(DevArray &&o) noexcept : p_(o.p_), n_(o.n_) {
    o.p_ = nullptr;
    o.n_ = 0;
  }
  DevArray &operator=(DevArray &&o) noexcept {
    if (this != &o) {
      release();
      p_ = o.p_;
      n_ = o.n_;
      o.p_ = nullptr;
      o.n_ = 0;
    }
    return *this;
  }
  ~DevArray() { release(); }
  // From the device cache; when the array is released (other than by an
  // exception), the work on its engine's stream that uses it must have been
  // waited for (engine members: the engine synchronises before destruction).
  void alloc(size_t n) {
    release();
    if (n) p_ = static_cast<T *>(DevicePool::take(n * sizeof(T)));
    n_ = n;
  }
  void upload(const std::vector<T> &v, cudaStream_t s) {
    alloc(v.size());
    if (n_) CK(cudaMemcpyAsync(p_, v.data(), n_ * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  T *get() const { return p_; }
  size_t size() const { return n_; }
  size_t bytes() const { return n_ * sizeof(T); }
  void release() {
    if (p_) DevicePool::put(p_);
    p_ = nullptr;
    n_ = 0;
  }

 private:
  T *p_ = nullptr;
  size_t n_ = 0;
};

}  // namespace agd
