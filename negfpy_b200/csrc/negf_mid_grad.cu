// Launches of the device-solve adjoint of orders up to 104 (negf_mid_adj.cuh).
#include "negf_mid_adj.cuh"
#include "negf_mid_launch.cuh"

namespace negf {
namespace mid {

int grad_grid(int np, int n, int L) {
  return with_adj(np, [&](auto c) { return slots_of<decltype(c)>(grad_ws<decltype(c)>(n, L)); });
}
size_t grad_ws_bytes(int np, int n, int L, int grid) {
  return with_adj(np, [&](auto c) { return (size_t)grid * grad_ws<decltype(c)>(n, L) * 16; });
}
int grad_launch(const GradArgs& ga, int np, int grid, double2* ws, cudaStream_t st) {
  return with_adj(np, [&](auto c) {
    using C = decltype(c);
    if (raise_smem<grad_kernel<C>, C>()) return -3;
    grad_kernel<C><<<grid < ga.r.batch ? grid : ga.r.batch, C::NTH, shared_bytes<C>(), st>>>(ga, ws);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace mid
}  // namespace negf
