// FP64 building blocks for one (omega, k) point of order 49..104 on one thread
// block: the matrix at work (a product's result, the matrix being inverted) in
// registers, one operand in shared memory, everything else in the block's
// global workspace (L2).
//
// At these orders a matrix is 83 KB (72) to 173 KB (104), so neither three of
// them fit shared memory nor does tiling through L2 keep the FP64 pipe busy:
// the kernels before this design read both operands of every 16 x 16 tile from
// L2/L1 and streamed the whole matrix through L2 in each of the n/8 updates of
// an inverse (45-51 % of the FP64 pipe at n = 96).  Here warp w owns row tile w
// (8 rows, every column): a product reads each row of its left operand from
// global memory once per block, straight into MMA fragments one chunk ahead,
// and its right operand from shared memory; the inverse (smem::gj_invert) keeps
// the matrix in registers throughout.  A row of a product's result belongs to
// the warp that needs it as the next left operand, so alpha g, U and the like
// pass through global memory without a block barrier.
#pragma once
#include "negf_common.cuh"
#include "negf_f64.h"
#include "negf_smem.cuh"

namespace negf {
namespace mid {

using smem::Acc;
using smem::AFrag;
using smem::Lane;
using smem::sidx;
using smem::z_of;

template <int NP, int OCC, int PARK>
using Cfg = smem::Cfg<NP, 1, NP / 8, OCC, 8, 2, PARK>;

template <class C>
struct Shared {
  smem::GJ<C> gj;
  double red[40];
  uint32_t tmem;
  int point;
};
template <class C>
constexpr size_t shared_bytes() { return (size_t)C::BUF * 16 + sizeof(Shared<C>); }

// A left operand in global memory: rows x cols elements, row stride ld; zero
// outside.
struct Left {
  const double2* p;
  int ld, rows, cols;
};

// Fragment (row r0 or, conjugate-transposed, column r0; k) of chunk kc.
template <bool CT>
__device__ __forceinline__ void load_left(AFrag& f, const Left& A, const Lane& L, int kc) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = kc * 8 + L.t + 4 * h;
    const bool in = CT ? (k < A.rows && L.r0 < A.cols) : (L.r0 < A.rows && k < A.cols);
    const double2 v = in ? (CT ? A.p[(long long)k * A.ld + L.r0] : A.p[(long long)L.r0 * A.ld + k])
                         : make_double2(0.0, 0.0);
    f.re[h] = v.x;
    f.im[h] = CT ? -v.y : v.y;
  }
}

// c = op(A) op(X), or c += with ADD: A from global memory, X in shared memory.  The next chunk's
// A and the next column tile's B are loaded under the current tile's MMAs.
template <class C, bool AC, bool BC, bool ADD = false>
__device__ __forceinline__ void prod(Acc<C>& c, const Left& A, const double2* X, int kch, const Lane& L) {
  int bb[2];
  smem::b_base<C, BC>(L, bb);
  if (!ADD) c.zero();
  AFrag a, an, b, bn;
  load_left<AC>(a, A, L, 0);
  smem::load_b<C, BC>(b, X, bb, 0, 0);
#pragma unroll 1
  for (int kc = 0; kc < kch; ++kc) {
    const int kn = kc + 1 < kch ? kc + 1 : 0;
    load_left<AC>(an, A, L, kn);
#pragma unroll
    for (int j = 0; j < C::TC; ++j) {
      if (j + 1 < C::TC) smem::load_b<C, BC>(bn, X, bb, kc, j + 1);
      else smem::load_b<C, BC>(bn, X, bb, kn, 0);
      smem::chunk(c.re[0][j], c.im[0][j], a, b);
      b = bn;
    }
    a = an;
  }
}

// Global nr x nc matrix (row stride ld) -> X, zeros outside.  The copies are
// complete for this thread on return; the caller's barrier publishes them.
template <class C>
__device__ __forceinline__ void load_x(double2* X, const double2* __restrict__ G, int ld, int nr, int nc) {
  for (int idx = threadIdx.x; idx < C::MAT; idx += C::NTH) {
    const int r = idx / C::NP, c = idx - r * C::NP;
    const bool in = r < nr && c < nc;
    const double2* src = in ? G + (long long)r * ld + c : G;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(X + sidx<C::NP>(r, c))), "l"(src),
                 "r"(in ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
// f(j, q, row, column) over the thread's elements; the loads of three tiles at a
// time are in flight (all of them at once would spill the accumulators).
template <class C, class F>
__device__ __forceinline__ void tiles(const Lane& L, F&& f) {
#pragma unroll
  for (int j = 0; j < C::TC; ++j) {
    if (j % 3 == 0) asm volatile("" ::: "memory");
#pragma unroll
    for (int q = 0; q < 2; ++q) f(j, q, L.r0, L.c0 + 8 * j + q);
  }
}
// The thread's elements of an n x n matrix, zeros outside.
template <class C>
__device__ __forceinline__ void load_tiles(Acc<C>& c, const double2* G, int n, const Lane& L) {
  tiles<C>(L, [&](int j, int q, int r, int cc) {
    c.set(0, j, q, r < n && cc < n ? G[r * n + cc] : make_double2(0.0, 0.0));
  });
}
// c = z - D - c [- S], identity in the padding.
template <class C>
__device__ __forceinline__ void minus_d(Acc<C>& c, const double2* D, const double2* S, double2 z, int n, const Lane& L) {
  tiles<C>(L, [&](int j, int q, int r, int cc) {
    const double2 d = r < n && cc < n ? D[r * n + cc] : make_double2(0.0, 0.0);
    c.set(0, j, q, csub(cneg(d), c.get(0, j, q)));
  });
  if (S)
    tiles<C>(L, [&](int j, int q, int r, int cc) {
      const double2 s = r < n && cc < n ? S[r * n + cc] : make_double2(0.0, 0.0);
      c.set(0, j, q, csub(c.get(0, j, q), s));
    });
  smem::each<C>(L, [&](int, int j, int q, int r, int cc) {
    if (r >= n || cc >= n) c.set(0, j, q, make_double2(r == cc ? 1.0 : 0.0, 0.0));
    else if (r == cc) c.set(0, j, q, cadd(c.get(0, j, q), z));
  });
}
// The thread's elements of a matrix -> row-major workspace (row stride NP).
template <class C>
__device__ __forceinline__ void store_rows(double2* G, const Acc<C>& c, const Lane& L) {
#pragma unroll
  for (int j = 0; j < C::TC; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) G[L.r0 * C::NP + L.c0 + 8 * j + q] = c.get(0, j, q);
}
// The warp's rows of X -> row-major workspace.  Ends with the warp synchronised: a
// lane writes other elements than those it owns, and the next step may read the
// rows as a left operand or element by element.
template <class C>
__device__ __forceinline__ void copy_rows(double2* G, const double2* X, const Lane& L) {
  for (int e = threadIdx.x & 31; e < 8 * C::NP; e += 32) {
    const int r = L.R0 + e / C::NP, c = e % C::NP;
    G[r * C::NP + c] = X[sidx<C::NP>(r, c)];
  }
  __syncwarp();
}

// ------------------------------------------------------------ Sancho-Rubio --
// Workspace: alpha, beta, alpha g, beta g (row-major), eps_s (each thread's
// elements together); eps in Tensor Memory.
template <class C>
struct Eps {
  static constexpr int kMat = C::TC * 8;                   // TMEM columns of a warp
  static constexpr int kPark = C::PARK * 8;
  static constexpr int kWarps = (C::NW + 3) / 4;           // warps that share a lane quarter
  static constexpr int kNeed = kWarps * (kMat + kPark);
  static constexpr int kCols = kNeed <= 128 ? 128 : kNeed <= 256 ? 256 : 512;
  static_assert(kNeed <= 512 && kCols * C::OCC <= 512, "TMEM columns");
};
template <class C>
constexpr size_t sr_ws() { return 5 * (size_t)C::MAT; }  // complex elements per block

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) sr_kernel(SrArgs a, double2* ws, unsigned* counter) {
  constexpr int NP = C::NP, MAT = C::MAT, TC = C::TC;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  const int n = a.n, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  double2* const AL = ws + (long long)blockIdx.x * sr_ws<C>();
  double2 *const BE = AL + MAT, *const AG = BE + MAT, *const BG = AG + MAT, *const ES = BG + MAT;
  if (tid < 32) umma::tmem_alloc(&sh.tmem, Eps<C>::kCols);
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t eps = sh.tmem + ((uint32_t)(tid >> 5 & 3) << 21) + (uint32_t)(tid >> 7) * (Eps<C>::kMat + Eps<C>::kPark);
  const double tol2 = a.tol * a.tol;
  const unsigned htol = (unsigned)__double2hiint(a.tol);
  const Left wsl{nullptr, NP, NP, NP};
  auto left = [&](const double2* p) { Left l = wsl; l.p = p; return l; };

  for (;;) {
    if (tid == 0) sh.point = (int)atomicAdd(counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= a.batch) break;
    const long long kset = a.kidx ? (long long)a.kidx[p] : 0;
    const double2* h00 = a.h00 + kset * a.lead_stride;
    const double2* h01 = a.h01 + kset * a.lead_stride;
    const double2* h10 = a.h10 ? a.h10 + kset * a.lead_stride : nullptr;
    const double w = a.omega[p];
    const double2 z = z_of(w, a.eta[p]);
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      double2 v[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = L.r0, c = L.c0 + 8 * j + q;
        const bool in = r < n && c < n;
        v[q] = in ? h00[r * n + c] : make_double2(0.0, 0.0);
        ES[(2 * j + q) * C::NTH + tid] = v[q];
        AL[r * NP + c] = in ? h01[r * n + c] : make_double2(0.0, 0.0);
        BE[r * NP + c] = in ? (h10 ? h10[r * n + c] : cconj(h01[c * n + r])) : make_double2(0.0, 0.0);
      }
      smem::tmem_put(eps + j * 8, v);
    }
    int status = kOk, it = 0;  // sweeps begun
    bool converged = false;
    Acc<C> c;
    auto element = [&](int j, int q, double2 x) {  // of z - x, identity in the padding
      const int r = L.r0, cc = L.c0 + 8 * j + q;
      if (r < n && cc < n) return (r == cc) ? csub(z, x) : cneg(x);
      return make_double2(r == cc ? 1.0 : 0.0, 0.0);
    };
    unsigned hi = 0u;  // largest high word of the sweep: non-finite from 0x7ff00000 on
    int big = 0;       // an element of the new alpha or beta of magnitude tol or more
    auto add_eps = [&]() {  // eps += c
      smem::tmem_stored();
      smem::tmem_tiles<TC>(eps, [&](int j, double2(&x)[2]) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          x[q] = cadd(x[q], c.get(0, j, q));
          hi = max(hi, smem::hi_word(x[q]));
        }
        smem::tmem_put(eps + j * 8, x);
      });
    };
    auto measure = [&]() {  // as in smem::sr_f64_kernel
      unsigned h = 0u;
      smem::each<C>(L, [&](int i, int j, int q, int, int) { h = max(h, smem::hi_word(c.get(i, j, q))); });
      hi = max(hi, h);
      if (h > htol) big = 1;
      else smem::each<C>(L, [&](int i, int j, int q, int, int) { big |= !(cabs2(c.get(i, j, q)) < tol2); });
    };
    for (;;) {
      // (z - eps)^-1, or the surface GF (z - eps_s)^-1 once converged
      if (!converged) {
        ++it;
        smem::tmem_stored();
        smem::tmem_tiles<TC>(eps, [&](int j, double2(&x)[2]) {
#pragma unroll
          for (int q = 0; q < 2; ++q) c.set(0, j, q, element(j, q, x[q]));
        });
      } else {
        tiles<C>(L, [&](int j, int q, int, int) { c.set(0, j, q, element(j, q, ES[(2 * j + q) * C::NTH + tid])); });
      }
      status = smem::gj_invert<C>(c, X, X, n, L, sh.gj, eps + Eps<C>::kMat);
      if (status != kOk || converged) break;
      prod<C, false, false>(c, left(AL), X, kch, L);  // alpha g
      store_rows<C>(AG, c, L);
      prod<C, false, false>(c, left(BE), X, kch, L);  // beta g
      store_rows<C>(BG, c, L);
      hi = 0u;
      big = 0;
      __syncthreads();
      load_x<C>(X, BE, NP, NP, NP);
      __syncthreads();
      prod<C, false, false>(c, left(AG), X, kch, L);  // (alpha g) beta
      tiles<C>(L, [&](int j, int q, int, int) {
        double2& e = ES[(2 * j + q) * C::NTH + tid];
        const double2 s = cadd(e, c.get(0, j, q));
        e = s;
        hi = max(hi, smem::hi_word(s));
      });
      add_eps();
      prod<C, false, false>(c, left(BG), X, kch, L);  // beta' = (beta g) beta; X keeps beta
      measure();
      store_rows<C>(BE, c, L);
      __syncthreads();
      load_x<C>(X, AL, NP, NP, NP);
      __syncthreads();
      prod<C, false, false>(c, left(BG), X, kch, L);  // (beta g) alpha
      add_eps();
      prod<C, false, false>(c, left(AG), X, kch, L);  // alpha' = (alpha g) alpha
      measure();
      store_rows<C>(AL, c, L);
      if (block_any(hi >= 0x7ff00000u)) {
        status = sr_failure_status(it, n, h00, h01, h10, z);
        break;
      }
      converged = !block_any(big);  // max(|alpha|, |beta|) < tol
      if (!converged && it == a.maxiter) {
        status = kMaxIter;
        break;
      }
    }
    if (status == kOk) {
      if (a.g_out) {
        double2* go = a.g_out + (long long)p * n * n;
        for (int idx = tid; idx < n * n; idx += C::NTH) {
          const int r = idx / n, cc = idx - r * n;
          go[idx] = X[sidx<NP>(r, cc)];
        }
      }
      if (a.dos_out) {
        // (omega/pi) Re Tr[i (g - g^H)] = (omega/pi) sum_j (-2 Im g_jj)
        double t = 0.0;
        for (int j = tid; j < n; j += C::NTH) t += -2.0 * X[sidx<NP>(j, j)].y;
        t = block_sum(t, sh.red);
        if (tid == 0) a.dos_out[p] = (w / 3.141592653589793238462643383279502884) * t;
      }
    } else if (a.dos_out && tid == 0) {
      a.dos_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
    }
    if (tid == 0) {
      if (a.iters_out) a.iters_out[p] = it;
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
  smem::tmem_stored();
  __syncthreads();
  if (tid < 32) umma::tmem_dealloc(sh.tmem, Eps<C>::kCols);
}

// ---------------------------------------------------------------- RGF sweep --
// Sigma = V g V^H into S (n x n); U is workspace, X is free before and after.
template <class C>
__device__ __forceinline__ void self_energy(double2* S, const double2* V, const double2* g, int n, int nl, double2* U,
                                            double2* X, const Lane& L) {
  const int lch = (nl + 7) >> 3;
  Acc<C> c;
  load_x<C>(X, g, nl, nl, nl);
  __syncthreads();
  prod<C, false, false>(c, Left{V, nl, n, nl}, X, lch, L);
  store_rows<C>(U, c, L);
  __syncthreads();
  load_x<C>(X, V, nl, n, nl);
  __syncthreads();
  prod<C, false, true>(c, Left{U, C::NP, C::NP, C::NP}, X, lch, L);
  smem::each<C>(L, [&](int i, int j, int q, int r, int cc) {
    if (r < n && cc < n) S[r * n + cc] = c.get(i, j, q);
  });
  __syncthreads();
}

// Element of Gamma = i (Sigma - Sigma^H), zero outside n x n.
__device__ __forceinline__ double2 gamma_of(const double2* S, int n, int r, int c) {
  if (r >= n || c >= n) return make_double2(0.0, 0.0);
  const double2 d = csub(S[r * n + c], cconj(S[c * n + r]));
  return make_double2(-d.y, d.x);
}

// T = Re sum_ij (Gamma_L G Gamma_R)_ij conj(G)_ij for G in the row-major
// workspace; GL, U: workspace.  The terms are summed as 8 warps walking 16 x 16
// tiles of the largest order nmax would (an order that does not depend on the
// padding or the split).
// Returns the sum in the first warp.
template <class C>
__device__ __forceinline__ double trace_t(const double2* sigL, const double2* sigR, const double2* G, double2* GL,
                                          double2* U, int n, int nmax, double2* X, double* red, const Lane& L) {
  constexpr int NP = C::NP;
  const int tid = threadIdx.x, kch = (n + 7) >> 3;
  Acc<C> c;
  tiles<C>(L, [&](int, int, int r, int cc) { GL[r * NP + cc] = gamma_of(sigL, n, r, cc); });
  __syncwarp();
  load_x<C>(X, G, NP, NP, NP);
  __syncthreads();
  const Left gl{GL, NP, NP, NP}, u{U, NP, NP, NP};
  prod<C, false, false>(c, gl, X, kch, L);
  store_rows<C>(U, c, L);
  __syncthreads();
  tiles<C>(L, [&](int, int, int r, int cc) { X[sidx<NP>(r, cc)] = gamma_of(sigR, n, r, cc); });
  __syncthreads();
  prod<C, false, false>(c, u, X, kch, L);
  __syncthreads();
  double* terms = reinterpret_cast<double*>(X);
  tiles<C>(L, [&](int j, int q, int r, int cc) {
    const double2 g = G[r * NP + cc];
    double t = 0.0;
    t += c.re[0][j][q] * g.x + c.im[0][j][q] * g.y;
    terms[r * NP + cc] = t;
  });
  __syncthreads();
  const int np16 = (nmax + 15) >> 4;
  for (int v = tid >> 5; v < 8; v += C::NW) {
    double t = 0.0;
    for (int s = v; s < np16 * np16; s += 8)
      for (int e = 0; e < 8; ++e) {
        const int r = (s / np16) * 16 + L.g + 8 * ((e >> 1) & 1), cc = (s % np16) * 16 + 8 * (e >> 2) + 2 * L.t + (e & 1);
        if (r < NP && cc < NP) t += terms[r * NP + cc];
      }
    t = warp_sum(t);
    if ((tid & 31) == 0) red[v] = t;
  }
  __syncthreads();
  return tid < 32 ? warp_sum(tid < 8 ? red[tid] : 0.0) : 0.0;
}

// Workspace: g, G_{0,l}, U (row-major), Sigma_L, Sigma_R.
template <class C>
constexpr size_t rgf_ws(int n) { return 3 * (size_t)C::MAT + 2 * (size_t)n * n; }

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) rgf_kernel(RgfArgs a, double2* ws) {
  static_assert(C::PARK == 0, "no Tensor Memory here");
  constexpr int NP = C::NP, MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  const int n = a.n, nlay = a.L, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  double2* const Gl = ws + (long long)blockIdx.x * rgf_ws<C>(n);
  double2 *const G0 = Gl + MAT, *const U = G0 + MAT, *const sigL = U + MAT, *const sigR = sigL + (long long)n * n;
  const Left gl{Gl, NP, NP, NP}, g0{G0, NP, NP, NP}, u{U, NP, NP, NP};

  for (;;) {
    if (tid == 0) sh.point = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= a.batch) break;
    const int lst = a.lead_status ? a.lead_status[p] : 0;
    if (lst != kOk) {
      if (tid == 0) {
        a.T_out[p] = __longlong_as_double(0x7ff8000000000000ULL);
        if (a.status_out) a.status_out[p] = lst;
      }
      continue;
    }
    const long long k = a.kidx ? (long long)a.kidx[p] : 0;
    const double2 z = z_of(a.omega[p], a.eta_dev[p]);
    const double2* D = a.D + k * a.d_ks;
    const double2* Cg = a.C + k * a.c_ks;
    self_energy<C>(sigL, a.VL + k * a.vl_ks, a.gL + (long long)p * a.gl_ps, n, a.nl, U, X, L);
    self_energy<C>(sigR, a.VR + k * a.vr_ks, a.gR + (long long)p * a.gr_ps, n, a.nr, U, X, L);
    Acc<C> c;
    int status = kOk;
    for (int l = 0; l < nlay; ++l) {
      if (l > 0) {
        // U = G_{0,l-1} C (own rows), W = g_{l-1} C into X
        const double2* Cl = Cg + (long long)(l - 1) * a.c_ls;
        __syncthreads();
        load_x<C>(X, Cl, n, n, n);
        __syncthreads();
        prod<C, false, false>(c, g0, X, kch, L);
        store_rows<C>(U, c, L);
        prod<C, false, false>(c, gl, X, kch, L);
        __syncthreads();
        smem::store_acc<C>(X, c, L);
        __syncthreads();
        prod<C, true, false>(c, Left{Cl, n, n, n}, X, kch, L);  // C^H W
      }
      // M = z - D_l - (C^H W, or Sigma_L on layer 0) [- Sigma_R on the last layer], identity padding
      if (l == 0) load_tiles<C>(c, sigL, n, L);
      minus_d<C>(c, D + (long long)l * a.d_ls, l == nlay - 1 ? sigR : nullptr, z, n, L);
      __syncthreads();  // every read of W is done
      status = smem::gj_invert<C>(c, X, X, n, L, sh.gj);
      if (status != kOk) break;
      // g_l, and G_{0,0} = g_0, G_{0,l} = U g_l
      if (l + 1 < nlay) copy_rows<C>(Gl, X, L);
      if (l == 0) {
        copy_rows<C>(G0, X, L);
      } else {
        prod<C, false, false>(c, u, X, kch, L);
        store_rows<C>(G0, c, L);
      }
    }
    __syncthreads();
    double tval = 0.0;
    if (status == kOk) {
      tval = trace_t<C>(sigL, sigR, G0, Gl, U, n, max(n, max(a.nl, a.nr)), X, sh.red, L);
      if (!isfinite(tval)) status = kNonFinite;
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

}  // namespace mid
}  // namespace negf
