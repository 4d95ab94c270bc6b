// Launches of the surface-GF adjoint of orders up to 104 (negf_mid_adj.cuh).
#include "negf_mid_adj.cuh"
#include "negf_mid_launch.cuh"

namespace negf {
namespace mid {

int sgf_adj_grid(int np) {
  return with_adj(np, [](auto c) { return grid_of<decltype(c)>(); });
}
size_t sgf_adj_ws_bytes(int np, int grid) {
  return with_adj(np, [&](auto c) { return (size_t)grid * sgf_adj_ws<decltype(c)>() * 16; });
}
int sgf_adj_launch(const SgfAdjArgs& sa, int np, int grid, double2* ws, cudaStream_t st) {
  return with_adj(np, [&](auto c) {
    using C = decltype(c);
    if (raise_smem<sgf_adjoint_kernel<C>, C>()) return -3;
    sgf_adjoint_kernel<C><<<grid < sa.batch ? grid : sa.batch, C::NTH, shared_bytes<C>(), st>>>(sa, ws);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace mid
}  // namespace negf
