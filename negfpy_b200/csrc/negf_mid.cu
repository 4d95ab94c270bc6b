// Instances and launches of the one-point-per-block kernels of order 49..104
// (negf_mid.cuh).
//
// Splits (thread blocks per SM, column tiles parked in the pivot steps) are the
// fastest of those measured.  1024 points, L = 20, decimation / device solve in
// ms: n = 54 9.2 / 7.2, n = 63 12.0 / 9.6, n = 72 21.3 / 16.3, n = 75 26.1 /
// 20.9, n = 84 32.5 / 25.5, n = 96 38.7 / 30.5.  Two blocks share an SM up to
// order 72 (83 KB of shared memory each); above, a second block does not fit.
// Parking tiles takes the pivot steps of the decimation from 745 to 600 cycles at
// n = 96 (spills); the device solve does not gain from it.
//
// Registers a thread follow from the warps a scheduler holds: 168 for three, 128
// for four, 96 for five, so orders 72 (two blocks of nine warps put five on one
// scheduler) and 104 (thirteen warps, four) spill where their neighbours hardly
// do.  Bytes stored / loaded a thread, decimation and device solve: 72 1676 / 1288
// and 1820 / 1860, 104 1428 / 1120 and 2144 / 2188; the other orders at most 40 / 56
// and 212 / 360.
#include "negf_mid_launch.cuh"

namespace negf {
namespace mid {

// f with the split of the padded order (56 .. 104).
template <class F>
static auto with_sr(int np, F&& f) {
  switch (np) {
    case 56: return f(Cfg<56, 2, 2>{});
    case 64: return f(Cfg<64, 2, 4>{});
    case 72: return f(Cfg<72, 2, 1>{});
    case 80: return f(Cfg<80, 1, 6>{});
    case 88: return f(Cfg<88, 1, 8>{});
    case 96: return f(Cfg<96, 1, 6>{});
    default: return f(Cfg<104, 1, 3>{});
  }
}
template <class F>
static auto with_rgf(int np, F&& f) {
  switch (np) {
    case 56: return f(Cfg<56, 2, 0>{});
    case 64: return f(Cfg<64, 2, 0>{});
    case 72: return f(Cfg<72, 2, 0>{});
    case 80: return f(Cfg<80, 1, 0>{});
    case 88: return f(Cfg<88, 1, 0>{});
    case 96: return f(Cfg<96, 1, 0>{});
    default: return f(Cfg<104, 1, 0>{});
  }
}

int sr_grid(int np) {
  return with_sr(np, [](auto c) { return grid_of<decltype(c)>(); });
}
int rgf_grid(int np) {
  return with_rgf(np, [](auto c) { return grid_of<decltype(c)>(); });
}
size_t sr_ws_bytes(int np, int grid) {
  return with_sr(np, [&](auto c) { return (size_t)grid * sr_ws<decltype(c)>() * 16; });
}
size_t rgf_ws_bytes(int np, int n, int grid) {
  return with_rgf(np, [&](auto c) { return (size_t)grid * rgf_ws<decltype(c)>(n) * 16; });
}
int sr_launch(const SrArgs& a, int np, int grid, double2* ws, unsigned* counter, cudaStream_t st) {
  if (a.batch <= 0) return 0;
  return with_sr(np, [&](auto c) {
    using C = decltype(c);
    if (raise_smem<sr_kernel<C>, C>()) return -3;
    sr_kernel<C><<<grid < a.batch ? grid : a.batch, C::NTH, shared_bytes<C>(), st>>>(a, ws, counter);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}
int rgf_launch(const RgfArgs& a, int np, int grid, double2* ws, cudaStream_t st) {
  if (a.batch <= 0) return 0;
  return with_rgf(np, [&](auto c) {
    using C = decltype(c);
    if (raise_smem<rgf_kernel<C>, C>()) return -3;
    rgf_kernel<C><<<grid < a.batch ? grid : a.batch, C::NTH, shared_bytes<C>(), st>>>(a, ws);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace mid
}  // namespace negf
