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
// Blocks of a kernel that keeps matrices of every layer: all that are resident at
// once while their workspace fits 512 MiB, else no more than two an SM, which
// bounds what a long device takes (full G, n = 32, 40 layers: 0.6 GB instead of
// 1.2).  Two cost the adjoint of 2368 points 1.17 times the time of four at n = 32
// and 1.46 at 16 (6 layers: 3.14 -> 3.68 ms, 0.76 -> 1.12), that of 296 nothing.
template <class C>
static int slots_of(size_t elems_per_block) {
  const int g = grid_of<C>();
  if (C::OCC <= 2 || g <= 0 || (size_t)g * elems_per_block * 16 <= ((size_t)512 << 20)) return g;
  return g / C::OCC * 2;
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

// f with the split of an adj_order() up to kMaxOrder: the padded orders of the
// decimation without 40, 56 and 88.  Those three are not built; orders 33..40,
// 49..56 and 81..88 run on the next split, and the missing ones would take 0.82,
// 0.86 and 0.90 of its time (adjoint, full G and surface-GF adjoint at 40, 56, 88
// against 48, 64, 96; 148 to 1184 points).
//
// Blocks per SM as for the decimation, four up to order 32.  Spills as there:
// the adjoint of the device solve stores / loads 5056 / 6580 bytes a thread at 72 and
// 5476 / 6160 at 104, 512 / 960 or less elsewhere; the full G 2044 / 2116 and
// 2324 / 2512, the surface-GF adjoint 1288 / 1616 and 1864 / 2108.
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
