// FP64 kernels of the per-(omega, k) phonon NEGF path.
//
//   smem::sr_f64_kernel   Sancho-Rubio decimation (negfpy core/surface_gf.py:18-81)
//                         with the surface DOS (core/dos.py:31-61), orders 2..48.
//   smem::rgf_f64_kernel  Sigma = V g V^H for both contacts (core/negf.py:72-97),
//                         left-connected recursive Green's function sweep for
//                         G_{0,L-1} of A = z - D - Sigma (core/negf.py:141-250,
//                         replacing the SuperLU solve at :353), Gamma = i(S - S^H)
//                         (:115-116) and T = Re Tr[Gamma_L G Gamma_R G^H] (:356).
//   *_scalar_kernel       the same for 1 x 1 blocks (the monatomic chain), one
//                         thread per point.
//   the reductions: k mean and moments, kappa, heat current, FCS cumulants.
#include <atomic>
#include <cstdio>

#include "negf_common.cuh"
#include "negf_f64.h"
#include "negf_smem.cuh"

namespace negf {

using smem::z_of;

// ------------------------------------------------------------ 1 x 1 blocks --
__global__ void sr_scalar_kernel(SrArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.batch) return;
  const long long k = a.kidx ? (long long)a.kidx[p] : 0;
  const double2 h00 = a.h00[k * a.lead_stride];
  const double2 h01 = a.h01[k * a.lead_stride];
  const double2 h10 = a.h10 ? a.h10[k * a.lead_stride] : cconj(h01);
  const double w = a.omega[p];
  const double2 z = z_of(w, a.eta[p]);
  double2 al = h01, be = h10, e = h00, es = h00;
  int status = kOk, it;
  bool conv = false;
  const double tol2 = a.tol * a.tol;
  for (it = 1; it <= a.maxiter; ++it) {
    const double2 m = csub(z, e);
    if (m.x == 0.0 && m.y == 0.0) { status = kSingular; break; }
    const double2 g = crecip(m);
    const double2 ag = cmul(al, g), bg = cmul(be, g);
    const double2 agb = cmul(ag, be), bga = cmul(bg, al);
    es = cadd(es, agb);
    e = cadd(cadd(e, agb), bga);
    al = cmul(ag, al);
    be = cmul(bg, be);
    if (!cfinite(es) || !cfinite(e) || !cfinite(al) || !cfinite(be)) {
      // as sr_failure_status, for one thread's 1 x 1 blocks
      const bool quiet = it == 1 && !(cfinite(h00) && cfinite(h01) && cfinite(h10) && cfinite(z));
      status = quiet ? kNonFinite : kUnstable;
      break;
    }
    if (fmax(cabs2(al), cabs2(be)) < tol2) { conv = true; break; }
  }
  if (status == kOk && !conv) { status = kMaxIter; it = a.maxiter; }
  double2 gs = make_double2(0.0, 0.0);
  if (status == kOk) {
    const double2 m = csub(z, es);
    if (m.x == 0.0 && m.y == 0.0) status = kSingular;
    else gs = crecip(m);
  }
  if (status == kOk && a.g_out) a.g_out[p] = gs;
  if (a.dos_out)
    a.dos_out[p] = (status == kOk) ? (w / 3.141592653589793238462643383279502884) * (-2.0 * gs.y)
                                   : __longlong_as_double(0x7ff8000000000000ULL);
  if (a.iters_out) a.iters_out[p] = it;
  if (a.status_out) a.status_out[p] = status;
}

__global__ void rgf_scalar_kernel(RgfArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.batch) return;
  const int lst = a.lead_status ? a.lead_status[p] : 0;
  if (lst != kOk) {
    a.T_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
    if (a.status_out) a.status_out[p] = lst;
    return;
  }
  const long long k = a.kidx ? (long long)a.kidx[p] : 0;
  const double2 z = z_of(a.omega[p], a.eta_dev[p]);
  const double2 vl = a.VL[k * a.vl_ks], vr = a.VR[k * a.vr_ks];
  const double2 sl = cmul(cmul(vl, a.gL[(long long)p * a.gl_ps]), cconj(vl));
  const double2 sr = cmul(cmul(vr, a.gR[(long long)p * a.gr_ps]), cconj(vr));
  const double2* D = a.D + k * a.d_ks;
  const double2* C = a.C + k * a.c_ks;
  const int L = a.L;
  int status = kOk;
  double2 m = csub(csub(z, D[0]), sl);
  if (L == 1) m = csub(m, sr);
  double2 g = make_double2(0.0, 0.0), g0 = g;
  if (m.x == 0.0 && m.y == 0.0) status = kSingular;
  else { g = crecip(m); g0 = g; }
  for (int l = 1; l < L && status == kOk; ++l) {
    const double2 c = C[(long long)(l - 1) * a.c_ls];
    const double2 w = cmul(g, c);
    const double2 u = cmul(g0, c);
    m = csub(csub(z, D[(long long)l * a.d_ls]), cmul(cconj(c), w));
    if (l == L - 1) m = csub(m, sr);
    if (m.x == 0.0 && m.y == 0.0) { status = kSingular; break; }
    g = crecip(m);
    g0 = cmul(u, g);
  }
  double t = 0.0;
  if (status == kOk) {
    // Gamma = i (S - S^*) = -2 Im(S) for 1 x 1 blocks
    const double gl = -2.0 * sl.y, gr = -2.0 * sr.y;
    t = gl * gr * cabs2(g0);
    if (!isfinite(t)) status = kNonFinite;
  }
  a.T_out[p] = (status == kOk) ? t : __longlong_as_double(0x7ff8000000000000ULL);
  if (a.status_out) a.status_out[p] = status;
}

// ------------------------------------------------------------- k-avg, kappa --
// tbar[w] = mean_k T[w, k] over points laid out omega-major (index w*K + k).
__global__ void kavg_kernel(const double* __restrict__ T, int W, int K, double* __restrict__ tbar) {
  const int w = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= W) return;
  double s = 0.0;
  for (int k = lane; k < K; k += 32) s += T[(long long)w * K + k];
  s = warp_sum(s);
  if (lane == 0) tbar[w] = s / (double)K;
}

// k moments <T> and <T^2> of an omega-major [W][K] table, one warp per omega
// (the moments of negfpy workflows/ifc_bulk.py:1690-1784).
__global__ void kmoments_kernel(const double* __restrict__ T, int W, int K, double* __restrict__ t1,
                                double* __restrict__ t2) {
  const int w = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= W) return;
  double s = 0.0, q = 0.0;
  for (int k = lane; k < K; k += 32) {
    const double v = T[(long long)w * K + k];
    s += v;
    q += v * v;
  }
  s = warp_sum(s);
  q = warp_sum(q);
  if (lane == 0) {
    t1[w] = s / (double)K;
    t2[w] = q / (double)K;
  }
}

// Heat-current cumulants from transmission moments (negfpy
// core/fcs.py:48-150), one block:
//   C1 = (1/2pi) trapz(<T> (A_L - A_R), w),
//   C2 = (1/2pi) trapz(<T> (B_L + B_R) + (<T> + <T^2>) (A_L - A_R)^2, w),
//   A = kB T phi1(x), B = (kB T)^2 phi2(x), x = hbar w / (kB T),
//   phi1 = x / expm1(x), phi2 = x^2 e^x / expm1(x)^2, with negfpy's series for
//   |x| < 1e-6 and 0 from x = 700 on.
__device__ __forceinline__ double fcs_phi1(double x) {
  if (fabs(x) < 1e-6) return 1.0 - 0.5 * x + (x * x) / 12.0 - (x * x * x * x) / 720.0;
  if (x < 700.0) return x / expm1(x);
  return 0.0;
}
__device__ __forceinline__ double fcs_phi2(double x) {
  if (fabs(x) < 1e-6) return 1.0 - (x * x) / 12.0 + (x * x * x * x) / 240.0;
  if (x < 700.0) {
    const double em1 = expm1(x);
    return (x * x) * (em1 + 1.0) / (em1 * em1);
  }
  return 0.0;
}
__global__ void fcs_kernel(const double* __restrict__ om, const double* __restrict__ t1, const double* __restrict__ t2,
                           int W, double temp_l, double temp_r, double* __restrict__ out) {
  __shared__ double red[40];
  const double hbar = 1.054571817e-34, kb = 1.380649e-23;
  const double sl = kb * temp_l, sr = kb * temp_r;
  double c1 = 0.0, c2 = 0.0;
  for (int i = threadIdx.x; i < W - 1; i += blockDim.x) {
    double f1[2], f2[2];
    for (int q = 0; q < 2; ++q) {
      const double w = om[i + q];
      const double xl = hbar * w / sl, xr = hbar * w / sr;
      const double ad = __dmul_rn(sl, fcs_phi1(xl)) - __dmul_rn(sr, fcs_phi1(xr));
      const double bs = sl * sl * fcs_phi2(xl) + sr * sr * fcs_phi2(xr);
      const double a = t1[i + q], b = t2[i + q];
      f1[q] = a * ad;
      f2[q] = a * bs + (a + b) * (ad * ad);
    }
    const double dw = om[i + 1] - om[i];
    c1 += dw * (f1[0] + f1[1]) / 2.0;
    c2 += dw * (f2[0] + f2[1]) / 2.0;
  }
  c1 = block_sum(c1, red);
  c2 = block_sum(c2, red);
  if (threadIdx.x == 0) {
    const double pref = 1.0 / (2.0 * 3.141592653589793238462643383279502884);
    out[0] = pref * c1;
    out[1] = pref * c2;
  }
}

// kappa(T) = (1/2pi) trapz(kB tbar(w) x^2 e^-x / (1 - e^-x)^2, w_rad), one
// block per temperature (negfpy workflows/ifc_bulk.py:408-438).
__global__ void kappa_kernel(const double* __restrict__ om, const double* __restrict__ tbar, int W,
                             const double* __restrict__ temps, double unit, double* __restrict__ out) {
  __shared__ double red[40];
  const double temp = temps[blockIdx.x];
  const double hbar = 1.054571817e-34, kb = 1.380649e-23;
  double s = 0.0;
  if (temp > 0.0) {
    for (int i = threadIdx.x; i < W - 1; i += blockDim.x) {
      double f[2];
      for (int q = 0; q < 2; ++q) {
        const double wr = om[i + q] * unit;
        const double x = hbar * wr / (kb * temp);
        double ker = 0.0;
        if (x < 1e-6) ker = 1.0 - x * x / 12.0;
        else if (x < 700.0) {
          const double y = exp(-x);
          const double d = 1.0 - y;
          ker = x * x * y / (d * d);
        }
        f[q] = kb * tbar[i + q] * ker;
      }
      s += (om[i + 1] * unit - om[i] * unit) * (f[0] + f[1]) / 2.0;
    }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[blockIdx.x] = (temp > 0.0) ? (1.0 / (2.0 * 3.141592653589793238462643383279502884)) * s : 0.0;
}

// Landauer heat current of each spectrum row b (block b):
//   J_b = (1/2pi) trapz((kB T_L phi(x_L) - kB T_R phi(x_R)) t_b(w), w),
//   phi(x) = x / expm1(x), x = hbar w / (kB T), with the series
//   1 - x/2 + x^2/12 below 1e-6 and 0 from 700 on (negfpy
//   core/thermal_current.py:30-67).
__device__ __forceinline__ double bose_phi(double x) {
  if (x < 1e-6) return 1.0 - 0.5 * x + (x * x) / 12.0;
  if (x < 700.0) return x / expm1(x);
  return 0.0;
}
__global__ void heat_current_kernel(const double* __restrict__ om, const double* __restrict__ t, int W, double temp_l,
                                    double temp_r, double* __restrict__ out) {
  __shared__ double red[40];
  const double hbar = 1.054571817e-34, kb = 1.380649e-23;
  const double* row = t + (long long)blockIdx.x * W;
  double s = 0.0;
  for (int i = threadIdx.x; i < W - 1; i += blockDim.x) {
    double f[2];
    for (int q = 0; q < 2; ++q) {
      const double w = om[i + q];
      // separately rounded products: equal temperatures cancel exactly
      const double wl = __dmul_rn(kb * temp_l, bose_phi(hbar * w / (kb * temp_l)));
      const double wr = __dmul_rn(kb * temp_r, bose_phi(hbar * w / (kb * temp_r)));
      f[q] = (wl - wr) * row[i + q];
    }
    s += (om[i + 1] - om[i]) * (f[0] + f[1]) / 2.0;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[blockIdx.x] = (1.0 / (2.0 * 3.141592653589793238462643383279502884)) * s;
}

// ---------------------------------------------------------------- launchers --
// Tile splits per padded order, the fastest of those measured (decimation /
// device solve of the same points, B200; the block before this design held one
// point in six shared buffers, padded to 16, 32 or 48):
//   48: 4 warps of 3 x 3 tiles, 2 points per SM.  4096 points, n = 48, L = 20:
//       17.5 / 16.0 ms (25.6 / 23.7 before); 12 warps of 1 x 3 20.7 / 18.7, 6 of
//       2 x 3 22.8 / 20.2.  Few fat warps win because the pivot steps of one
//       point share the FP64 pipe with the products of the other: each step's
//       instructions wait behind fewer queued MMAs.  Orders 33..40 pad to 48
//       as well: 40 (25 tiles, 5 warps) leaves two schedulers with half the
//       work, 15.6 / 13.6 against 14.6 / 13.2 ms at n = 36.
//   32: 4 warps of 2 x 2, 4 points.  4096 points, n = 30: 5.7 / 5.0 ms.
//   24: 3 warps of 1 x 3, 6 points.  9216 points, n = 24, L = 30: 6.8 / 8.9 ms
//       (12.9 / 21.0 before, padded to 32).
//   16: 2 warps of 1 x 2, 10 points; few points: 4 warps of one tile (see
//       kFewPoints16).
//   8:  1 warp, 16 points.
using C48 = smem::Cfg<48, 3, 3, 2>;
using C32 = smem::Cfg<32, 2, 2, 4>;
using C24 = smem::Cfg<24, 1, 3, 6>;
using C16 = smem::Cfg<16, 1, 2, 10>;
using C16Few = smem::Cfg<16, 1, 1, 4>;
using C8 = smem::Cfg<8, 1, 1, 16>;

// Last launch failure of this host thread (read by the C-ABI layer).
thread_local char g_launch_err[256] = "";

template <typename K>
static int record_failure(const char* what, K kernel, cudaError_t e, size_t smem, int threads) {
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, kernel);
  snprintf(g_launch_err, sizeof(g_launch_err),
           "%s: %s (threads %d, dynamic smem %zu, regs %d, max threads %d, static smem %zu)", what,
           cudaGetErrorString(e), threads, smem, fa.numRegs, fa.maxThreadsPerBlock, fa.sharedSizeBytes);
  return -3;
}

const char* last_launch_error() { return g_launch_err; }

// The dynamic shared memory limit of a kernel, raised once per device.
template <class C>
static int raise_smem(void (*kernel)(SrArgs)) {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return 0;
  const size_t sm = smem::shared_bytes<C>();
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return record_failure("sr_f64 smem attribute", kernel, e, sm, C::NTH);
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return 0;
}

template <class C>
static int launch_sr(const SrArgs& a, cudaStream_t st) {
  if (const int rc = raise_smem<C>(smem::sr_f64_kernel<C>)) return rc;
  const size_t sm = smem::shared_bytes<C>();
  smem::sr_f64_kernel<C><<<a.batch, C::NTH, sm, st>>>(a);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : record_failure("sr_f64 launch", smem::sr_f64_kernel<C>, e, sm, C::NTH);
}

// Blocks of the device solve that are resident at once on the current device
// (its persistent grid), or negative on error.
template <class C>
static int grid_rgf() {
  static std::atomic<int> grid[64];
  int dev = 0;
  cudaGetDevice(&dev);
  const int known = dev < 64 ? grid[dev].load(std::memory_order_acquire) : 0;
  if (known > 0) return known;
  const size_t sm = smem::shared_bytes<C>();
  const cudaError_t e =
      cudaFuncSetAttribute(smem::rgf_f64_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return record_failure("rgf_f64 smem attribute", smem::rgf_f64_kernel<C>, e, sm, C::NTH);
  int per = 0, nsm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, smem::rgf_f64_kernel<C>, C::NTH, sm) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per <= 0)
    return -3;
  if (dev < 64) grid[dev].store(per * nsm, std::memory_order_release);
  return per * nsm;
}

template <class C>
static int launch_rgf(const RgfArgs& a, int grid, cudaStream_t st) {
  const int own = grid_rgf<C>();
  if (own < 0) return own;
  if (grid > own) grid = own;
  if (grid > a.batch) grid = a.batch;
  const size_t sm = smem::shared_bytes<C>();
  smem::rgf_f64_kernel<C><<<grid, C::NTH, sm, st>>>(a);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : record_failure("rgf_f64 launch", smem::rgf_f64_kernel<C>, e, sm, C::NTH);
}

// Padded size for an order-n block: 1 (scalar path), 8, 16, 24, 32 or 48.
int padded_order(int n) {
  if (n == 1) return 1;
  if (n <= 32) return (n + 7) / 8 * 8;
  if (n <= 48) return 48;
  return 0;
}

// Up to this many points of order 9..16 (four blocks of C16Few per SM at once)
// latency counts, and one tile per warp is faster: n = 12, L = 30, decimation +
// device solve 247 us against 327 for 148 points, 328 against 385 for 324, 394
// against 414 for 592; 645 against 582 for 900.
constexpr int kFewPoints16 = 592;

int sr_f64_launch(const SrArgs& a, cudaStream_t st) {
  if (a.batch <= 0) return 0;
  switch (padded_order(a.n)) {
    case 1: {
      const int tpb = 128;
      sr_scalar_kernel<<<(a.batch + tpb - 1) / tpb, tpb, 0, st>>>(a);
      return cudaGetLastError() == cudaSuccess ? 0 : -3;
    }
    case 8: return launch_sr<C8>(a, st);
    case 16: return a.batch <= kFewPoints16 ? launch_sr<C16Few>(a, st) : launch_sr<C16>(a, st);
    case 24: return launch_sr<C24>(a, st);
    case 32: return launch_sr<C32>(a, st);
    case 48: return launch_sr<C48>(a, st);
    default: return -2;
  }
}

// The largest persistent grid of any split of the order (sizes the scratch).
int rgf_f64_grid(int np) {
  switch (np) {
    case 1: return 0;
    case 8: return grid_rgf<C8>();
    case 16: {
      const int a = grid_rgf<C16>(), b = grid_rgf<C16Few>();
      return a < 0 || b < 0 ? -3 : (a > b ? a : b);
    }
    case 24: return grid_rgf<C24>();
    case 32: return grid_rgf<C32>();
    case 48: return grid_rgf<C48>();
    default: return -2;
  }
}

int rgf_f64_launch(const RgfArgs& a, int np, int grid, cudaStream_t st) {
  if (a.batch <= 0) return 0;
  switch (np) {
    case 1: {
      const int tpb = 128;
      rgf_scalar_kernel<<<(a.batch + tpb - 1) / tpb, tpb, 0, st>>>(a);
      return cudaGetLastError() == cudaSuccess ? 0 : -3;
    }
    case 8: return launch_rgf<C8>(a, grid, st);
    case 16: return a.batch <= kFewPoints16 ? launch_rgf<C16Few>(a, grid, st) : launch_rgf<C16>(a, grid, st);
    case 24: return launch_rgf<C24>(a, grid, st);
    case 32: return launch_rgf<C32>(a, grid, st);
    case 48: return launch_rgf<C48>(a, grid, st);
    default: return -2;
  }
}

int kavg_launch(const double* T, int W, int K, double* tbar, cudaStream_t st) {
  if (W <= 0) return 0;
  const int wpb = 8;
  kavg_kernel<<<(W + wpb - 1) / wpb, wpb * 32, 0, st>>>(T, W, K, tbar);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int kmoments_launch(const double* T, int W, int K, double* t1, double* t2, cudaStream_t st) {
  if (W <= 0) return 0;
  const int wpb = 8;
  kmoments_kernel<<<(W + wpb - 1) / wpb, wpb * 32, 0, st>>>(T, W, K, t1, t2);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int fcs_launch(const double* om, const double* t1, const double* t2, int W, double temp_l, double temp_r, double* out,
               cudaStream_t st) {
  fcs_kernel<<<1, 256, 0, st>>>(om, t1, t2, W, temp_l, temp_r, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int heat_current_launch(const double* om, const double* t, int W, int n_spectra, double temp_l, double temp_r,
                        double* out, cudaStream_t st) {
  if (n_spectra <= 0) return 0;
  heat_current_kernel<<<n_spectra, 256, 0, st>>>(om, t, W, temp_l, temp_r, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int kappa_launch(const double* om, const double* tbar, int W, const double* temps, int nT, double unit, double* out,
                 cudaStream_t st) {
  if (nT <= 0) return 0;
  kappa_kernel<<<nT, 256, 0, st>>>(om, tbar, W, temps, unit, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace negf
