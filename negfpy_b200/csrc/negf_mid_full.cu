// Launches of the full device Green's function of orders up to 104
// (negf_mid_adj.cuh): rounds of at most `grid` points, sweep and diagonal first,
// then the walks.
#include "negf_mid_adj.cuh"
#include "negf_mid_launch.cuh"

namespace negf {
namespace mid {

int full_grid(int np, int n, int L) {
  return with_adj(np, [&](auto c) { return slots_of<decltype(c)>(full_ws<decltype(c)>(n, L)); });
}
size_t full_ws_bytes(int np, int n, int L, int grid) {
  return with_adj(np, [&](auto c) { return (size_t)grid * full_ws<decltype(c)>(n, L) * 16; });
}
int full_launch(const FullArgs& fa, int np, int grid, double2* ws, cudaStream_t st) {
  return with_adj(np, [&](auto c) {
    using C = decltype(c);
    if (raise_smem<full_diag_kernel<C>, C>() || raise_smem<full_walk_kernel<C>, C>()) return -3;
    for (int first = 0; first < fa.r.batch; first += grid) {
      const int pts = fa.r.batch - first < grid ? fa.r.batch - first : grid;
      full_diag_kernel<C><<<pts, C::NTH, shared_bytes<C>(), st>>>(fa, first, ws);
      if (fa.r.L > 1)
        full_walk_kernel<C><<<pts * 2 * (fa.r.L - 1), C::NTH, shared_bytes<C>(), st>>>(fa, first, ws);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace mid
}  // namespace negf
