// Uneven batch: many independent lead/device/lead systems of different block
// orders, layer counts and k grids in one call of persistent kernels.
//
// A work item is (system, k index, omega).  Each block takes items from an
// atomic counter in the order the host gave them (largest estimated cost
// first, so the tail of the launch is short), and runs for its item:
//   1. the left lead's Sancho-Rubio decimation at the lead's own padded order
//      (negfpy core/surface_gf.py:18-81), and the right lead's unless the
//      system's leads are the same,
//   2. the device solve at the system's padded order, in FP64
//      (rgf_point_f64) or with the FP32 sweep (rgf_point_mixed),
// writing T, the status and the decimation sweeps of the item.  Block orders
// up to 256; the per-block workspace and the shared memory are sized for the
// largest order in the batch.
//
// In FP64 with orders above kSplit in the batch, those items run first in a kernel
// of their own on the strips of negf_big.cuh (one block per SM, which two blocks
// of the other kernel cannot join), and the kernel for the rest is launched as
// its programmatic dependent: its blocks take the SMs as the first kernel's run
// out of items, so the short items still fill the tail of the long ones.
// 240 items of order 192 among 648 of 24..120: 236 -> 204 ms.
#include <atomic>

#include "../../include/negf_b200.h"
#include "negf_big.cuh"
#include "negf_common.cuh"
#include "negf_f64.h"
#include "negf_mixed.cuh"
#include "negf_point.cuh"
#include "negf_tiles.cuh"

namespace negf {
namespace batch {

using glob::kThreads;

struct BatchArgs {
  const NegfBatchSystem* sys;
  int n_systems;
  const int* item_system;
  const int* item_k;
  const double* item_omega;
  int n_items;
  double tol;
  int maxiter;
  double* T_out;
  int* status_out;
  int* iters_out;
  unsigned* counter;
  int big_order;   // items of order kSplit + 1 .. big_order run in big_kernel (0: none)
  bool dependent;  // launched as the other kernel's programmatic dependent
};
// The largest order that stays with the smaller items.  One block an SM: the strips
// are faster from 129 on (135 and 144: 0.91-0.97 of the time).  Two: at 129..144
// the second block hides more than the strips save (ms, strips / two blocks: 296
// items of order 144 67.2 / 64.8, 520 of 135 122.6 / 115.6), above not (296 items
// of 150 74.7 / 81.4, of 192 115.5 / 145.5).
template <int MINB>
constexpr int kSplit = MINB == 2 ? 144 : 128;

__host__ __device__ inline int pad16(int n) { return (n + 15) / 16 * 16; }
// Per-block workspace, in complex128 elements, for padded order NP: the two
// compact lead surface GFs and the scratch of the larger of the decimation
// (7 NP^2), the FP64 device solve (6 NP^2 + 2 n^2) and the mixed one
// (7 NP^2 + 2 n^2 in complex128 units).
__host__ __device__ inline size_t block_elems(int np) { return 2 * (size_t)np * np + 9 * (size_t)np * np; }

__device__ __forceinline__ bool bad_item(const NegfBatchSystem& d, long long k, int order) {
  const int n = d.n_dev, nl = d.n_lead_l, nr = d.n_lead_r;
  return k < 0 || k >= d.n_k || n <= 0 || nl <= 0 || nr <= 0 || d.n_layers <= 0 || n > order || nl > order ||
         nr > order || (d.same_leads && nl != nr);
}

// MINB: blocks per SM the register allocation is capped for (1: no cap,
// 2: at most 128 registers a thread, with some spilling).
template <bool MIXED, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) batch_kernel(BatchArgs a, int NPmax, double2* ws) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* red = reinterpret_cast<double*>(smraw + ((glob::gjs_bytes(NPmax) + 15) / 16) * 16);
  __shared__ int s_item;
  const int tid = threadIdx.x;
  const long long M2max = (long long)NPmax * NPmax;
  double2* base = ws + (long long)blockIdx.x * block_elems(NPmax);
  double2* gl = base;
  double2* gr = base + M2max;
  double2* scratch = base + 2 * M2max;

  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int p = s_item;
    __syncthreads();
    if (p >= a.n_items) break;
    const int si = a.item_system[p];
    if (si < 0 || si >= a.n_systems) {
      if (tid == 0) {
        a.T_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
        if (a.status_out) a.status_out[p] = kBadItem;
        if (a.iters_out) a.iters_out[p] = 0;
      }
      continue;
    }
    const NegfBatchSystem& d = a.sys[si];
    const long long k = a.item_k[p];
    const double w = a.item_omega[p];
    const int n = d.n_dev, nl = d.n_lead_l, nr = d.n_lead_r;
    const int top = max(n, max(nl, nr));
    if (top > kSplit<MINB> && top <= a.big_order) continue;
    int status = bad_item(d, k, NPmax) ? kBadItem : kOk, iters = 0;
    // 1. lead surface GFs (compact, row stride = lead order)
    for (int side = 0; side < 2 && status == kOk; ++side) {
      if (side == 1 && d.same_leads) break;
      const int m = side ? nr : nl;
      const int NPl = pad16(m);
      const glob::GJS sh = glob::carve(smraw, NPl);
      const long long ks = side ? d.lead_r_kstride : d.lead_l_kstride;
      const double2* h00 = reinterpret_cast<const double2*>(side ? d.lead_r_h00 : d.lead_l_h00) + k * ks;
      const double2* h01 = reinterpret_cast<const double2*>(side ? d.lead_r_h01 : d.lead_l_h01) + k * ks;
      const double* h10r = side ? d.lead_r_h10 : d.lead_l_h10;
      const double2* h10 = h10r ? reinterpret_cast<const double2*>(h10r) + k * ks : nullptr;
      int it = 0;
      double2* pg = nullptr;
      status = glob::sr_point(m, NPl, h00, h01, h10, glob::z_of(w, d.eta), a.tol, a.maxiter, scratch, sh, red,
                              &it, &pg);
      if (side == 0) iters = it;
      if (status == kOk) {
        double2* dst = side ? gr : gl;
        for (int e = tid; e < m * m; e += kThreads) {
          const int r = e / m, c = e - r * m;
          dst[e] = pg[(long long)r * NPl + c];
        }
      }
      __syncthreads();
    }
    // 2. device solve
    double tval = 0.0;
    if (status == kOk) {
      const int NP = pad16(max(n, max(nl, nr)));
      glob::RgfPoint q;
      q.n = n;
      q.nl = nl;
      q.nr = nr;
      q.L = d.n_layers;
      q.D = reinterpret_cast<const double2*>(d.onsite) + k * d.onsite_kstride;
      q.d_ls = d.onsite_lstride;
      q.C = reinterpret_cast<const double2*>(d.coupling ? d.coupling : d.onsite) + k * d.coupling_kstride;
      q.c_ls = d.coupling_lstride;
      q.VL = reinterpret_cast<const double2*>(d.v_left) + k * d.v_left_kstride;
      q.VR = reinterpret_cast<const double2*>(d.v_right) + k * d.v_right_kstride;
      q.gL = gl;
      q.gR = d.same_leads ? gl : gr;
      q.z = glob::z_of(w, d.eta_device);
      if (MIXED) {
        const mixed::GJS32 sh = mixed::carve32(smraw, NP);
        status = mixed::rgf_point_mixed(q, NP, reinterpret_cast<unsigned char*>(scratch), sh, red, &tval);
      } else {
        const glob::GJS sh = glob::carve(smraw, NP);
        status = glob::rgf_point_f64(q, NP, scratch, sh, red, &tval);
      }
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
      if (a.iters_out) a.iters_out[p] = iters;
    }
    __syncthreads();
  }
  // The launch is complete when the kernel before it is, too.
  if (a.dependent && blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Decimation and solve in one loop spill more than in kernels of their own: 224 /
// 564 bytes a thread (stored / loaded) up to order 192, 1064 / 3912 above, against
// 28 / 52 and 248 / 340 of big::sr_kernel and 0 and 200 / 464 of big::rgf_kernel.
//
// The items of order SPLIT + 1 .. a.big_order.  Workspace per block: the lead
// surface GFs and the scratch of the decimation (7 NP^2; the device solve needs
// less).
__host__ __device__ inline size_t big_elems(int np) { return 9 * (size_t)np * np; }
template <int NT, int SPLIT>
__global__ void __launch_bounds__(NT, 1) big_kernel(BatchArgs a, int NPmax, double2* ws) {
  extern __shared__ __align__(16) unsigned char smraw[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  big::Ctl& sh = *reinterpret_cast<big::Ctl*>(smraw + big::region_bytes<2>(NPmax));
  const int tid = threadIdx.x;
  double2* const gl = ws + (long long)blockIdx.x * big_elems(NPmax);
  double2 *const gr = gl + NPmax * NPmax, *const scratch = gr + NPmax * NPmax;
  for (;;) {
    if (tid == 0) sh.point = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= a.n_items) break;
    const int si = a.item_system[p];
    if (si < 0 || si >= a.n_systems) continue;
    const NegfBatchSystem& d = a.sys[si];
    const int top = max(d.n_dev, max(d.n_lead_l, d.n_lead_r));
    if (top <= SPLIT || top > a.big_order) continue;
    const long long k = a.item_k[p];
    const double w = a.item_omega[p];
    int status = bad_item(d, k, a.big_order) ? kBadItem : kOk, iters = 0;
#pragma unroll 1
    for (int side = 0; side < 2 && status == kOk; ++side) {
      if (side == 1 && d.same_leads) break;
      const int m = side ? d.n_lead_r : d.n_lead_l;
      const big::Geo G(pad16(m));
      const long long ks = k * (side ? d.lead_r_kstride : d.lead_l_kstride);
      const double2* h00 = reinterpret_cast<const double2*>(side ? d.lead_r_h00 : d.lead_l_h00) + ks;
      const double2* h01 = reinterpret_cast<const double2*>(side ? d.lead_r_h01 : d.lead_l_h01) + ks;
      const double* h10r = side ? d.lead_r_h10 : d.lead_l_h10;
      const double2* h10 = h10r ? reinterpret_cast<const double2*>(h10r) + ks : nullptr;
      int it = 0;
      double2* g = nullptr;
      status = big::sr_point<2>(m, G, h00, h01, h10, big::z_of(w, d.eta), a.tol, a.maxiter, scratch, smraw, sh, &it, &g);
      if (side == 0) iters = it;
      if (status == kOk) {
        double2* dst = side ? gr : gl;
        for (int e = tid; e < m * m; e += G.nthr) dst[e] = g[e / m * G.NP + e % m];
      }
      __syncthreads();
    }
    double tval = 0.0;
    if (status == kOk) {
      const big::Geo G(pad16(top));
      const big::Point q{d.n_dev, d.n_lead_l, d.n_lead_r, d.n_layers,
                         reinterpret_cast<const double2*>(d.onsite) + k * d.onsite_kstride, d.onsite_lstride,
                         reinterpret_cast<const double2*>(d.coupling ? d.coupling : d.onsite) + k * d.coupling_kstride,
                         d.coupling_lstride, reinterpret_cast<const double2*>(d.v_left) + k * d.v_left_kstride,
                         reinterpret_cast<const double2*>(d.v_right) + k * d.v_right_kstride, gl,
                         d.same_leads ? gl : gr, big::z_of(w, d.eta_device)};
      status = big::rgf_point<2>(q, G, scratch, smraw, sh, &tval);
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
      if (a.iters_out) a.iters_out[p] = iters;
    }
    __syncthreads();
  }
}

size_t smem_bytes(int npmax) { return ((glob::gjs_bytes(npmax) + 15) / 16) * 16 + 40 * 8; }

// Largest dynamic shared memory already configured per (device, variant):
// the attribute is set once, outside any stream capture that replays the launch.
std::atomic<int> g_smem_set[4][64];

template <bool MIXED, int MINB>
int configure(int npmax) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  const int sm = (int)smem_bytes(npmax);
  std::atomic<int>& cur = g_smem_set[(MIXED ? 2 : 0) + (MINB - 1)][dev];
  if (cur.load() >= sm) return 0;
  if (cudaFuncSetAttribute(batch_kernel<MIXED, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) !=
      cudaSuccess)
    return -3;
  cur.store(sm);
  return 0;
}

template <bool MIXED, int MINB>
int max_grid(int npmax) {
  if (configure<MIXED, MINB>(npmax) != 0) return -3;
  int nb = 0, dev = 0, nsm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_kernel<MIXED, MINB>, kThreads, smem_bytes(npmax)) !=
          cudaSuccess ||
      nb <= 0)
    return -3;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nb * nsm;
}

template <bool MIXED, int MINB>
int launch_variant(const BatchArgs& a, int npmax, int grid, double2* ws, cudaStream_t st) {
  if (configure<MIXED, MINB>(npmax) != 0) return -3;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = kThreads;
  cfg.dynamicSmemBytes = smem_bytes(npmax);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = a.dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, batch_kernel<MIXED, MINB>, a, npmax, ws) == cudaSuccess ? 0 : -3;
}

template <int NT, int SPLIT>
int launch_big(const BatchArgs& a, int npmax, int grid, double2* ws, cudaStream_t st) {
  static std::atomic<bool> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (!done[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(big_kernel<NT, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)big::shared_bytes<2>(NT / 2)) != cudaSuccess)
      return -3;
    done[dev].store(true, std::memory_order_release);
  }
  big_kernel<NT, SPLIT><<<grid, 2 * npmax, big::shared_bytes<2>(npmax), st>>>(a, npmax, ws);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// Blocks of the two kernels of an FP64 batch with orders above kSplit<MINB>.
struct Split {
  int big, rest;
};
template <int MINB>
Split split_grids(int grid) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int gmax = max_grid<false, MINB>(kSplit<MINB>);
  return {grid < nsm ? grid : nsm, grid < gmax ? grid : gmax};
}
template <int MINB>
size_t split_elems(const Split& g, int npmax) {
  return g.big * big_elems(npmax) + g.rest * block_elems(kSplit<MINB>);
}
// Their launches; 1 when the workspace is too small for both (one kernel then
// takes every item).  The counters are neighbours, both zero.
template <int MINB>
int launch_split(BatchArgs a, int npmax, int grid, double2* ws, size_t ws_bytes, cudaStream_t st) {
  const Split g = split_grids<MINB>(grid);
  if (g.big <= 0 || g.rest <= 0) return -3;
  if (split_elems<MINB>(g, npmax) * 16 > ws_bytes) return 1;
  a.big_order = npmax;
  const int rc = npmax <= 192 ? launch_big<384, kSplit<MINB>>(a, npmax, g.big, ws, st)
                              : launch_big<512, kSplit<MINB>>(a, npmax, g.big, ws, st);
  if (rc != 0) return rc;
  a.counter += 1;
  a.dependent = true;
  return launch_variant<false, MINB>(a, kSplit<MINB>, g.rest, ws + g.big * big_elems(npmax), st);
}

}  // namespace batch

int batch_max_grid(int npmax, int mixed, int minb) {
  if (minb == 2) return mixed ? batch::max_grid<true, 2>(npmax) : batch::max_grid<false, 2>(npmax);
  return mixed ? batch::max_grid<true, 1>(npmax) : batch::max_grid<false, 1>(npmax);
}
size_t batch_ws_bytes(int npmax, int grid) { return (size_t)grid * batch::block_elems(npmax) * 16; }
size_t batch_split_ws_bytes(int npmax, int mixed, int minb, int grid) {
  if (mixed || npmax <= (minb == 2 ? batch::kSplit<2> : batch::kSplit<1>)) return 0;
  return 16 * (minb == 2 ? batch::split_elems<2>(batch::split_grids<2>(grid), npmax)
                         : batch::split_elems<1>(batch::split_grids<1>(grid), npmax));
}
int batch_launch(const NegfBatchSystem* sys, int n_systems, const int* item_system, const int* item_k, const double* item_omega,
                 int n_items, double tol, int maxiter, double* t_out, int* status_out, int* iters_out, int npmax,
                 int mixed, int minb, int grid, void* counter, void* ws, size_t ws_bytes, cudaStream_t st) {
  batch::BatchArgs a;
  a.sys = sys;
  a.n_systems = n_systems;
  a.item_system = item_system;
  a.item_k = item_k;
  a.item_omega = item_omega;
  a.n_items = n_items;
  a.tol = tol;
  a.maxiter = maxiter;
  a.T_out = t_out;
  a.status_out = status_out;
  a.iters_out = iters_out;
  a.counter = static_cast<unsigned*>(counter);
  a.big_order = 0;
  a.dependent = false;
  double2* w = static_cast<double2*>(ws);
  if (!mixed && npmax > (minb == 2 ? batch::kSplit<2> : batch::kSplit<1>)) {
    const int rc = minb == 2 ? batch::launch_split<2>(a, npmax, grid, w, ws_bytes, st)
                             : batch::launch_split<1>(a, npmax, grid, w, ws_bytes, st);
    if (rc <= 0) return rc;
  }
  if (minb == 2)
    return mixed ? batch::launch_variant<true, 2>(a, npmax, grid, w, st)
                 : batch::launch_variant<false, 2>(a, npmax, grid, w, st);
  return mixed ? batch::launch_variant<true, 1>(a, npmax, grid, w, st)
               : batch::launch_variant<false, 1>(a, npmax, grid, w, st);
}

}  // namespace negf
