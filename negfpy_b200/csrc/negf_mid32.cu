// Launches of the mixed and the refined device solve for padded orders 16..96
// (negf_mid32.cuh); orders above and the tcgen05 products take the kernels of
// negf_mixed.cu and negf_refine.cu.
#include "negf_f64.h"
#include "negf_mid32.cuh"
#include "negf_mid_launch.cuh"

namespace negf {
namespace mid {

// Blocks per SM: as many as registers allow before the products spill badly; each
// block's phases leave units idle that another's use (n = 48, 888 points, 20
// layers: three blocks 11.6 ms, two 12.8; n = 63, 1776 points, 8 layers: two 17.9,
// one 22.4).  Orders 80 and 96: shared memory allows one or two, registers one.
// The refined solve still spills 1452 / 1460 bytes a thread (stored / loaded) at 48
// and 1240 / 1260 at 96, the mixed one 568 / 644 and 676 / 684.
template <class F>
static auto with32(int np, F&& f) {
  switch (np) {
    case 16: return f(Cfg<16, 8, 0>{});
    case 32: return f(Cfg<32, 5, 0>{});
    case 48: return f(Cfg<48, 3, 0>{});
    case 64: return f(Cfg<64, 2, 0>{});
    case 80: return f(Cfg<80, 1, 0>{});
    default: return f(Cfg<96, 1, 0>{});
  }
}
// Blocks that are resident at once and fit the workspace, no more than points: a
// block without one may start before another SM's, and its neighbour would then
// take a second point while that SM idles (148 points, 6 layers, mixed: n = 24
// 0.224 -> 0.125 ms, n = 32 0.280 -> 0.149).
template <class C>
static int fit(int batch, size_t per_block, size_t ws_bytes) {
  const int g = grid_of<C>();
  const size_t m = ws_bytes / per_block;
  const int f = m < (size_t)g ? (int)m : g;
  return f < batch ? f : batch;
}

size_t mixed32_ws_bytes(int np, int n) {
  return with32(np, [&](auto c) {
    using C = decltype(c);
    return (size_t)grid_of<C>() * mixed_ws_bytes<C>(n);
  });
}
size_t refine32_ws_bytes(int np, int n, int L) {
  return with32(np, [&](auto c) {
    using C = decltype(c);
    return (size_t)grid_of<C>() * refine_ws_bytes<C>(n, L);
  });
}
int mixed32_launch(const RgfArgs& a, int np, void* ws, size_t ws_bytes, cudaStream_t st) {
  return with32(np, [&](auto c) {
    using C = decltype(c);
    const int grid = fit<C>(a.batch, mixed_ws_bytes<C>(a.n), ws_bytes);
    if (grid <= 0 || raise_smem<mixed_kernel<C>, C>() != 0) return -3;
    mixed_kernel<C><<<grid, C::NTH, shared32_bytes<C>(), st>>>(a, static_cast<unsigned char*>(ws));
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}
int refine32_launch(const RgfArgs& a, int np, void* ws, size_t ws_bytes, double tol, int maxit, int* steps_out,
                    cudaStream_t st) {
  return with32(np, [&](auto c) {
    using C = decltype(c);
    const int grid = fit<C>(a.batch, refine_ws_bytes<C>(a.n, a.L), ws_bytes);
    if (grid <= 0 || raise_smem<refine_kernel<C>, C>() != 0) return -3;
    refine_kernel<C><<<grid, C::NTH, shared32_bytes<C>(), st>>>(a, static_cast<unsigned char*>(ws), tol, maxit,
                                                                 steps_out);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace mid
}  // namespace negf
