// Device memory of the library's buffers: a stream-ordered pool per device
// for what is built inside a PoolScope, cudaMalloc / cudaFree for the rest.
#include <mutex>

#include "dg_common.cuh"

namespace dg {
namespace {

constexpr int kMaxDevices = 64;

struct ScopeState {
  cudaStream_t stream = nullptr;
  bool on = false;
};
thread_local ScopeState t_scope;
thread_local size_t t_largest = 0;  // no limit

// The pool of a device, made on first use and kept for the process (its
// unused memory is bounded by kPoolKeep); nullptr where pools are not
// supported.
cudaMemPool_t device_pool(int dev) {
  static std::mutex mu;
  static cudaMemPool_t pools[kMaxDevices] = {};
  static bool tried[kMaxDevices] = {};
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!tried[dev]) {
    tried[dev] = true;
    int ok = 0;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    uint64_t keep = kPoolKeep;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess || !ok ||
        cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) {
      (void)cudaGetLastError();
      pools[dev] = nullptr;
    } else {
      cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  return pools[dev];
}

}  // namespace

// A small block allocated and freed.  Another one is kept per device, so that
// the 2 MB they lie in stay mapped: 5 us (cudaDeviceSynchronize 3; 600 with the
// mapping undone each time).
cudaError_t drain_device() {
  static std::mutex mu;
  static void* kept[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  constexpr size_t kSmall = 256;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev < kMaxDevices && !kept[dev] && cudaMalloc(&kept[dev], kSmall) != cudaSuccess) kept[dev] = nullptr;
  }
  void* p = nullptr;
  e = cudaMalloc(&p, kSmall);
  if (e == cudaSuccess) e = cudaFree(p);
  if (e == cudaErrorMemoryAllocation) e = wait_device();
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

std::shared_mutex& capture_lock() {
  static std::shared_mutex mu;
  return mu;
}
cudaError_t wait_device() {
  std::unique_lock<std::shared_mutex> lock(capture_lock());
  return cudaDeviceSynchronize();
}

PoolScope::PoolScope(cudaStream_t s) : prev_(t_scope.stream), prev_on_(t_scope.on) {
  t_scope.stream = s;
  t_scope.on = true;
}
PoolScope::~PoolScope() {
  t_scope.stream = prev_;
  t_scope.on = prev_on_;
}

cudaError_t device_alloc(void** p, size_t bytes, int* dev) {
  *p = nullptr;
  *dev = -1;
  if (t_largest && bytes > t_largest) return cudaErrorMemoryAllocation;
  int cur = 0;
  cudaError_t e = cudaGetDevice(&cur);
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = t_scope.on ? device_pool(cur) : nullptr;
  for (int attempt = 0; attempt < 2; ++attempt) {
    e = pool ? cudaMallocFromPoolAsync(p, bytes, pool, t_scope.stream) : cudaMalloc(p, bytes);
    if (e == cudaSuccess) {
      if (pool) *dev = cur;
      return e;
    }
    (void)cudaGetLastError();
    *p = nullptr;
    if (e != cudaErrorMemoryAllocation || attempt) break;
    // what the pool holds unused may be what is missing
    cudaMemPool_t held = device_pool(cur);
    if (!held || drain_device() != cudaSuccess || cudaMemPoolTrimTo(held, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      break;
    }
  }
  return e;
}

void device_free(void* p, int dev) {
  if (dev < 0) {
    cudaFree(p);
    return;
  }
  int cur = dev;
  cudaGetDevice(&cur);
  if (cur == dev && t_scope.on) {
    cudaFreeAsync(p, t_scope.stream);
    return;
  }
  // outside a scope (or with another device current): any stream may still use it
  if (cur != dev) cudaSetDevice(dev);
  if (drain_device() == cudaSuccess) cudaFreeAsync(p, nullptr);
  if (cur != dev) cudaSetDevice(cur);
}

}  // namespace dg

extern "C" dg_status dg_set_allocation_limit(int64_t bytes) {
  dg::t_largest = bytes > 0 ? size_t(bytes) : 0;
  return DG_OK;
}
