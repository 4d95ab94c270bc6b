// Decimation and device solve of orders 105..256 (negf_big.cuh): persistent
// blocks of np / 16 warps, each taking points from an atomic counter.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "negf_big.cuh"

namespace negf {
namespace big {

template <int NT, int OCC>
__global__ void __launch_bounds__(NT, OCC) sr_kernel(SrArgs a, int NP, double2* ws, unsigned* counter) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Ctl& sh = *reinterpret_cast<Ctl*>(smraw + region_bytes<3 - OCC>(NP));
  const Geo G(NP);
  const int n = a.n;
  double2* const W = ws + (long long)blockIdx.x * 7 * NP * NP;
  for (;;) {
    if (G.tid == 0) sh.point = (int)atomicAdd(counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= a.batch) break;
    const long long k = (a.kidx ? (long long)a.kidx[p] : 0) * a.lead_stride;
    const double w = a.omega[p];
    int it = 0;
    double2* g = nullptr;
    const int status = sr_point<3 - OCC>(n, G, a.h00 + k, a.h01 + k, a.h10 ? a.h10 + k : nullptr, z_of(w, a.eta[p]), a.tol,
                                a.maxiter, W, smraw, sh, &it, &g);
    if (status == kOk) {
      if (a.g_out) {
        double2* go = a.g_out + (long long)p * n * n;
        for (int e = G.tid; e < n * n; e += G.nthr) go[e] = g[e / n * NP + e % n];
      }
      if (a.dos_out) {
        // (omega/pi) Re Tr[i (g - g^H)] = (omega/pi) sum_j (-2 Im g_jj), summed as 256 threads would
        double t = 0.0;
        for (int j = G.tid; j < n; j += 256) t += -2.0 * g[j * NP + j].y;
        t = block_sum(G.tid < 256 ? t : 0.0, sh.red);
        if (G.tid == 0) a.dos_out[p] = (w / 3.141592653589793238462643383279502884) * t;
      }
    } else if (a.dos_out && G.tid == 0) {
      a.dos_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
    }
    if (G.tid == 0) {
      if (a.iters_out) a.iters_out[p] = it;
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

template <int NT, int OCC>
__global__ void __launch_bounds__(NT, OCC) rgf_kernel(RgfArgs a, int NP, double2* ws) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Ctl& sh = *reinterpret_cast<Ctl*>(smraw + region_bytes<3 - OCC>(NP));
  const Geo G(NP);
  double2* const W = ws + (long long)blockIdx.x * rgf_elems(NP, a.n);
  for (;;) {
    if (G.tid == 0) sh.point = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= a.batch) break;
    const int lst = a.lead_status ? a.lead_status[p] : 0;
    if (lst != kOk) {
      if (G.tid == 0) {
        a.T_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
        if (a.status_out) a.status_out[p] = lst;
      }
      continue;
    }
    const long long k = a.kidx ? (long long)a.kidx[p] : 0;
    const Point q{a.n, a.nl, a.nr, a.L, a.D + k * a.d_ks, a.d_ls, a.C + k * a.c_ks, a.c_ls, a.VL + k * a.vl_ks,
                  a.VR + k * a.vr_ks, a.gL + (long long)p * a.gl_ps, a.gR + (long long)p * a.gr_ps,
                  z_of(a.omega[p], a.eta_dev[p])};
    double t = 0.0;
    const int status = rgf_point<3 - OCC>(q, G, W, smraw, sh, &t);
    if (G.tid == 0) {
      a.T_out[p] = (status == kOk) ? t : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

static int sms() {
  static std::atomic<int> known[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int n = dev < 64 ? known[dev].load(std::memory_order_acquire) : 0;
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (dev < 64) known[dev].store(n, std::memory_order_release);
  }
  return n;
}
// Two blocks an SM where their panels and factors fit (128 rows), which hides
// one's pivot steps behind the other's products; one above, and one for no more
// points than SMs (n = 105, 148 points: 25.2 -> 17.0 ms for the decimation, the two-block form spilling at its 128 registers).
// The register limit follows from the block size.
template <class F>
static auto with(int np, bool few, F&& f) {
  if (np <= 128 && few) return f(std::integral_constant<int, 256>{}, std::integral_constant<int, 1>{});
  if (np <= 128) return f(std::integral_constant<int, 256>{}, std::integral_constant<int, 2>{});
  if (np <= 192) return f(std::integral_constant<int, 384>{}, std::integral_constant<int, 1>{});
  return f(std::integral_constant<int, 512>{}, std::integral_constant<int, 1>{});
}
// The kernel's dynamic shared memory limit, raised to the most any order of its
// class needs, once per device.
template <auto kernel>
static int raise_smem(size_t bytes) {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return -3;
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return 0;
}

int grid(int np) {
  const int n = sms();
  if (n <= 0) return -3;
  return with(np, false, [&](auto, auto occ) { return n * decltype(occ)::value; });
}
size_t sr_ws_bytes(int np, int grid) { return (size_t)grid * 7 * np * np * 16; }
size_t rgf_ws_bytes(int np, int n, int grid) { return (size_t)grid * rgf_elems(np, n) * 16; }
int sr_launch(const SrArgs& a, int np, int grid, double2* ws, unsigned* counter, cudaStream_t st) {
  return with(np, a.batch <= sms(), [&](auto nt, auto occ) {
    constexpr int NT = decltype(nt)::value, OCC = decltype(occ)::value;
    if (raise_smem<sr_kernel<NT, OCC>>(shared_bytes<3 - OCC>(NT / 2)) != 0) return -3;
    sr_kernel<NT, OCC><<<OCC == 1 ? std::min(grid, sms()) : grid, 2 * np, shared_bytes<3 - OCC>(np), st>>>(a, np, ws, counter);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}
int rgf_launch(const RgfArgs& a, int np, int grid, double2* ws, cudaStream_t st) {
  return with(np, a.batch <= sms(), [&](auto nt, auto occ) {
    constexpr int NT = decltype(nt)::value, OCC = decltype(occ)::value;
    if (raise_smem<rgf_kernel<NT, OCC>>(shared_bytes<3 - OCC>(NT / 2)) != 0) return -3;
    rgf_kernel<NT, OCC><<<OCC == 1 ? std::min(grid, sms()) : grid, 2 * np, shared_bytes<3 - OCC>(np), st>>>(a, np, ws);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  });
}

}  // namespace big
}  // namespace negf
