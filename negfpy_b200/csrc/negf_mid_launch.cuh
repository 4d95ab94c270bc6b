// Host-side helpers of the launches in negf_mid*.cu.
#pragma once
#include <atomic>

#include "negf_mid.cuh"

namespace negf {
namespace mid {

// Blocks resident at once on the current device (from the split's budget: the
// occupancy query does not count Tensor Memory), or negative on error.
template <class C>
static int grid_of() {
  static std::atomic<int> sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int n = dev < 64 ? sms[dev].load(std::memory_order_acquire) : 0;
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -3;
    if (dev < 64) sms[dev].store(n, std::memory_order_release);
  }
  return n * C::OCC;
}
// The kernel's dynamic shared memory limit, raised once per device.
template <auto kernel, class C>
static int raise_smem() {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared_bytes<C>()) != cudaSuccess)
    return -3;
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return 0;
}

// f with the split of an adj_order() up to kMaxOrder.
template <class F>
static auto with_adj(int np, F&& f) {
  switch (np) {
    case 16: return f(Cfg<16, 4, 0>{});
    case 24: return f(Cfg<24, 4, 0>{});
    case 32: return f(Cfg<32, 4, 0>{});
    case 48: return f(Cfg<48, 2, 0>{});
    case 64: return f(Cfg<64, 2, 0>{});
    case 72: return f(Cfg<72, 2, 0>{});
    case 80: return f(Cfg<80, 1, 0>{});
    case 96: return f(Cfg<96, 1, 0>{});
    default: return f(Cfg<104, 1, 0>{});
  }
}

}  // namespace mid
}  // namespace negf
