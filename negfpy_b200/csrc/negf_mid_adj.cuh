// Adjoints of the device solve and of the lead surface GFs, and the full device
// Green's function, for orders up to 104 on the building blocks of
// negf_mid.cuh: a product's right operand in shared memory (X), its result and
// the matrix being inverted in registers, everything else in the block's global
// workspace (row-major, row stride NP).
#pragma once
#include "negf_mid.cuh"

namespace negf {
namespace mid {

// X <- a global nr x nc matrix / the block's result; the leading barrier ends
// every use of X and publishes the stores before it.
template <class C>
__device__ __forceinline__ void fill(double2* X, const double2* src, int ld, int nr, int nc) {
  __syncthreads();
  load_x<C>(X, src, ld, nr, nc);
  __syncthreads();
}
template <class C>
__device__ __forceinline__ void fill(double2* X, const double2* ws) {
  fill<C>(X, ws, C::NP, C::NP, C::NP);
}
template <class C>
__device__ __forceinline__ void fill(double2* X, const Acc<C>& c, const Lane& L) {
  __syncthreads();
  smem::store_acc<C>(X, c, L);
  __syncthreads();
}
template <class C>
__device__ __forceinline__ Left ws_left(const double2* p) {
  return Left{p, C::NP, C::NP, C::NP};
}
// Inverse of c into the workspace slot (X is scratch and holds it afterwards).
template <class C>
__device__ __forceinline__ int invert_to(double2* slot, Acc<C>& c, int n, double2* X, smem::GJ<C>& gj, const Lane& L) {
  __syncthreads();
  const int st = smem::gj_invert<C>(c, X, X, n, L, gj);
  if (st == kOk) copy_rows<C>(slot, X, L);
  return st;
}
__device__ __forceinline__ void atomic_cadd(double2* dst, double2 v) {
  atomicAdd(&dst->x, v.x);
  atomicAdd(&dst->y, v.y);
}
// A point's contribution to a gradient block: added atomically into the
// shared per-k block, or stored into the point's own block (per-point mode,
// which the host then sums in a fixed order for a reproducible result).
__device__ __forceinline__ void grad_put(double2* dst, double2 v, bool own) {
  if (own) *dst = v;
  else atomic_cadd(dst, v);
}

// ------------------------------------------------------- adjoint (gradient) --
// Per point: T and the weighted adjoint blocks of dT/dD.  With G = A^-1 for
// A = z - D - Sigma_L - Sigma_R, Y = Gamma_R G_{0,L-1}^H Gamma_L and
// X_{ji} = G_{j,L-1} Y G_{0,i},
//     dT = 2 Re sum_ij Tr[dD_ij X_ji],
// so a change dD_i of onsite block i contributes 2 Re Tr[dD_i X_ii] and a
// change dC_i of the coupling between layers i and i+1 (with dC_i^H below the
// diagonal) contributes 2 Re Tr[dC_i (X_{i+1,i} + X_{i,i+1}^H)].  The kernel
// adds weight[p] X_ii into grad_d[k][i] and weight[p] (X_{i+1,i} + X_{i,i+1}^H)
// into grad_c[k][i].  Nothing is kept from the forward pass: the left sweep
// (g^L), the last block column G_{j,L-1} (backward recursion), the right sweep
// (g^R) and the first block row G_{0,i} are recomputed here, per point.
// Workspace: 11 + 2 L matrices, Sigma_L and Sigma_R (n x n).
template <class C>
constexpr size_t grad_ws(int n, int L) { return (11 + 2 * (size_t)L) * C::MAT + 2 * (size_t)n * n; }

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) grad_kernel(GradArgs ga, double2* ws) {
  constexpr int NP = C::NP, MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  const RgfArgs& a = ga.r;
  const int n = a.n, nlay = a.L, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  double2* const base = ws + (long long)blockIdx.x * grad_ws<C>(n, nlay);
  double2 *const Y = base, *const Tt = base + MAT, *const Xb = base + 2 * MAT, *const GL = base + 3 * MAT,
          *const GR = base + 4 * MAT, *const Zl = base + 5 * MAT, *const Zr = base + 6 * MAT;
  double2* const gl = base + 11 * MAT;               // g^L_j, then G_{j,L-1}
  double2* const gr = gl + (long long)nlay * MAT;    // g^R_i
  double2* const sigL = gr + (long long)nlay * MAT;
  double2* const sigR = sigL + (long long)n * n;

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
    const double wgt = ga.weight[p];
    const bool own = ga.per_point != 0;
    const long long slot = own ? (long long)p : k;
    double2* gdk = ga.grad_d + slot * (long long)nlay * n * n;
    double2* gck = ga.grad_c + slot * (long long)(nlay > 1 ? nlay - 1 : 1) * n * n;
    double2 *Ap = base + 7 * MAT, *Ac = base + 8 * MAT, *G0p = base + 9 * MAT, *G0c = base + 10 * MAT;
    auto Dl = [&](int l) { return D + (long long)l * a.d_ls; };
    auto Cl = [&](int l) { return Left{Cg + (long long)l * a.c_ls, n, n, n}; };
    auto fill_c = [&](int l) { fill<C>(X, Cl(l).p, n, n, n); };
    Acc<C> c;

    self_energy<C>(sigL, a.VL + k * a.vl_ks, a.gL + (long long)p * a.gl_ps, n, a.nl, Tt, X, L);
    self_energy<C>(sigR, a.VR + k * a.vr_ks, a.gR + (long long)p * a.gr_ps, n, a.nr, Tt, X, L);
    tiles<C>(L, [&](int, int, int r, int cc) {
      GL[r * NP + cc] = gamma_of(sigL, n, r, cc);
      GR[r * NP + cc] = gamma_of(sigR, n, r, cc);
    });

    int status = kOk;
    // 1. left sweep: gl[l] = g^L_l
    for (int l = 0; l < nlay && status == kOk; ++l) {
      if (l == 0) {
        load_tiles<C>(c, sigL, n, L);
      } else {
        fill_c(l - 1);
        prod<C, false, false>(c, ws_left<C>(gl + (l - 1) * MAT), X, kch, L);
        fill<C>(X, c, L);
        prod<C, true, false>(c, Cl(l - 1), X, kch, L);
      }
      minus_d<C>(c, Dl(l), l == nlay - 1 ? sigR : nullptr, z, n, L);
      status = invert_to<C>(gl + l * MAT, c, n, X, sh.gj, L);
    }
    // 2. last block column: G_{L-1,L-1} = g^L_{L-1}, G_{j,L-1} = g^L_j C_j G_{j+1,L-1}
    for (int j = nlay - 2; j >= 0 && status == kOk; --j) {
      fill<C>(X, gl + (j + 1) * MAT);
      prod<C, false, false>(c, Cl(j), X, kch, L);
      fill<C>(X, c, L);
      prod<C, false, false>(c, ws_left<C>(gl + j * MAT), X, kch, L);
      store_rows<C>(gl + j * MAT, c, L);
    }
    double tval = 0.0;
    if (status == kOk) {
      // T = Re Tr[Gamma_L G Gamma_R G^H], G = G_{0,L-1};  Y = Gamma_R G^H Gamma_L
      fill<C>(X, gl);
      prod<C, false, false>(c, ws_left<C>(GL), X, kch, L);
      store_rows<C>(Tt, c, L);
      fill<C>(X, GR);
      prod<C, false, false>(c, ws_left<C>(Tt), X, kch, L);
      __syncthreads();
      // the terms summed as 256 threads striding over the rows of the matrix
      // padded to a multiple of 16 would
      double* terms = reinterpret_cast<double*>(X);
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        const double2 g = gl[r * NP + cc];
        double t = 0.0;
        t += c.re[0][j][q] * g.x + c.im[0][j][q] * g.y;
        terms[r * NP + cc] = t;
      });
      __syncthreads();
      const int np16 = (max(n, max(a.nl, a.nr)) + 15) / 16 * 16;
      for (int v = tid >> 5; v < 8; v += C::NW) {
        double t = 0.0;
        for (int e = v * 32 + (tid & 31); e < np16 * np16; e += 256) {
          const int r = e / np16, cc = e - r * np16;
          if (r < n && cc < n) t += terms[r * NP + cc];
        }
        t = warp_sum(t);
        if ((tid & 31) == 0) sh.red[v] = t;
      }
      __syncthreads();
      tval = warp_sum((tid & 31) < 8 ? sh.red[tid & 31] : 0.0);
      if (!isfinite(tval)) status = kNonFinite;
      fill<C>(X, GL);
      prod<C, true, false>(c, ws_left<C>(gl), X, kch, L);
      fill<C>(X, c, L);
      prod<C, false, false>(c, ws_left<C>(GR), X, kch, L);
      store_rows<C>(Y, c, L);
    }
    // 3. right sweep: gr[i] = g^R_i, then G_{0,0}
    for (int i = nlay - 1; i >= 0 && status == kOk; --i) {
      if (i == nlay - 1) {
        load_tiles<C>(c, sigR, n, L);
      } else {
        fill<C>(X, gr + (i + 1) * MAT);
        prod<C, false, false>(c, Cl(i), X, kch, L);
        store_rows<C>(Tt, c, L);
        fill_c(i);
        prod<C, false, true>(c, ws_left<C>(Tt), X, kch, L);
      }
      minus_d<C>(c, Dl(i), i == 0 ? sigL : nullptr, z, n, L);
      status = invert_to<C>(i == 0 ? G0c : gr + i * MAT, c, n, X, sh.gj, L);
    }
    // Contact terms of dT/dSigma: Sigma_L enters A_00 (like D_00) and Gamma_L,
    // so dT/dSigma_L = X_00 + i G Gamma_R G^H; likewise dT/dSigma_R =
    // X_{L-1,L-1} + i G^H Gamma_L G, with G = G_{0,L-1} (slot 0 of gl).
    const bool want_l = ga.sig_adj_l != nullptr, want_r = ga.sig_adj_r != nullptr;
    if (status == kOk && want_l) {
      fill<C>(X, GR);
      prod<C, false, false>(c, ws_left<C>(gl), X, kch, L);
      store_rows<C>(Tt, c, L);
      fill<C>(X, gl);
      prod<C, false, true>(c, ws_left<C>(Tt), X, kch, L);
      store_rows<C>(Zl, c, L);
    }
    if (status == kOk && want_r) {
      fill<C>(X, GL);
      prod<C, true, false>(c, ws_left<C>(gl), X, kch, L);
      store_rows<C>(Tt, c, L);
      fill<C>(X, gl);
      prod<C, false, false>(c, ws_left<C>(Tt), X, kch, L);
      store_rows<C>(Zr, c, L);
    }
    // 4. first block row and the adjoint blocks
    for (int i = 0; i < nlay && status == kOk; ++i) {
      fill<C>(X, Y);
      prod<C, false, false>(c, ws_left<C>(gl + i * MAT), X, kch, L);
      store_rows<C>(Ac, c, L);
      fill<C>(X, G0c);
      if (i >= 1) {
        prod<C, false, false>(c, ws_left<C>(Ap), X, kch, L);  // X_{i-1,i}
        store_rows<C>(Xb, c, L);
      }
      prod<C, false, false>(c, ws_left<C>(Ac), X, kch, L);  // X_{i,i}
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        if (r < n && cc < n) {
          const double2 v = c.get(0, j, q);
          grad_put(gdk + (long long)i * n * n + r * n + cc, make_double2(wgt * v.x, wgt * v.y), own);
          if (i == 0 && want_l) {
            const double2 zt = Zl[r * NP + cc];
            ga.sig_adj_l[(long long)p * n * n + r * n + cc] = make_double2(wgt * (v.x - zt.y), wgt * (v.y + zt.x));
          }
          if (i == nlay - 1 && want_r) {
            const double2 zt = Zr[r * NP + cc];
            ga.sig_adj_r[(long long)p * n * n + r * n + cc] = make_double2(wgt * (v.x - zt.y), wgt * (v.y + zt.x));
          }
        }
      });
      if (i >= 1) {
        fill<C>(X, G0p);
        prod<C, false, false>(c, ws_left<C>(Ac), X, kch, L);  // X_{i,i-1}
        tiles<C>(L, [&](int j, int q, int r, int cc) {
          if (r < n && cc < n) {
            const double2 v = cadd(c.get(0, j, q), cconj(Xb[cc * NP + r]));
            grad_put(gck + (long long)(i - 1) * n * n + r * n + cc, make_double2(wgt * v.x, wgt * v.y), own);
          }
        });
      }
      if (i + 1 < nlay) {
        fill_c(i);
        prod<C, false, false>(c, ws_left<C>(G0c), X, kch, L);
        store_rows<C>(Tt, c, L);
        fill<C>(X, gr + (i + 1) * MAT);
        prod<C, false, false>(c, ws_left<C>(Tt), X, kch, L);  // G_{0,i+1} into the spare buffer
        store_rows<C>(G0p, c, L);
        double2* t = G0p;
        G0p = G0c;
        G0c = t;
        t = Ap;
        Ap = Ac;
        Ac = t;
      }
    }
    __syncthreads();
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

// ------------------------------------------------ adjoint of the surface GF --
// Per point, with the surface GF g of the lead (negfpy core/surface_gf.py:18-81
// computes it by decimation) and the weighted adjoint X of Sigma = V g V^H
// from grad_kernel (dT = 2 Re Tr[dSigma X]):
//
//   gbar = V^H X V,   Vbar = g V^H X + g^H V^H X^H            (dT = 2 Re Tr[dV Vbar])
//
// g solves g = (z - H00 - H01 g H10)^-1, so with P = g H01 and Q = H10 g,
//   dg - P dg Q = g (dH00 + dH01 g H10 + H01 g dH10) g,
// and Tr[dg gbar] = Tr[(dH00 + dH01 g H10 + H01 g dH10) g Lam g] where Lam
// solves the transposed equation Lam - Q Lam P = gbar.  Lam = sum_k Q^k gbar P^k
// is summed by doubling (Smith's method): Lam += A Lam B, A <- A^2, B <- B^2
// from A = Q, B = P, until max(max|A|, max|B|) < tol; no inverse is needed and
// nothing is differentiated through the decimation sweeps.  Then
//   H00bar = g Lam g,  H01bar = g H10 H00bar,  H10bar = H00bar H01 g,
// added into the per-k accumulators (with H10 = H01^H, H10bar^H is added to
// H01bar instead).  Status: kMaxIter if the doubling does not converge within
// maxiter, kNonFinite on inf/nan.  Workspace: 7 matrices.
template <class C>
constexpr size_t sgf_adj_ws() { return 7 * (size_t)C::MAT; }

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) sgf_adjoint_kernel(SgfAdjArgs sa, double2* ws) {
  constexpr int NP = C::NP, MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  const int nl = sa.nl, n = sa.n, tid = threadIdx.x;
  const int kl = (nl + 7) >> 3, kd = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  double2* const base = ws + (long long)blockIdx.x * sgf_adj_ws<C>();
  double2 *const T1 = base, *const T2 = base + MAT, *const Lam = base + 2 * MAT, *const Tt = base + 3 * MAT,
          *const Aq = base + 4 * MAT, *const Bp = base + 5 * MAT, *const U = base + 6 * MAT;

  for (;;) {
    if (tid == 0) sh.point = (int)atomicAdd(sa.counter, 1u);
    __syncthreads();
    const int p = sh.point;
    __syncthreads();
    if (p >= sa.batch) break;
    const int lst = sa.lead_status ? sa.lead_status[p] : 0;
    if (lst != kOk) {
      if (tid == 0) {
        if (sa.status_out) sa.status_out[p] = lst;
        if (sa.iters_out) sa.iters_out[p] = 0;
      }
      continue;
    }
    const long long k = sa.kidx ? (long long)sa.kidx[p] : 0;
    const double2* h01 = sa.h01 + k * sa.lead_stride;
    const double2* h10 = sa.h10 ? sa.h10 + k * sa.lead_stride : nullptr;
    const double2* V = sa.V + k * sa.v_ks;
    const double2* xs = sa.xs + (long long)p * n * n;
    const double2* g = sa.g + (long long)p * sa.g_ps;
    const Left lv{V, nl, n, nl}, lx{xs, n, n, n}, lg{g, nl, nl, nl}, lh01{h01, nl, nl, nl}, lh10{h10, nl, nl, nl};
    const bool own = sa.per_point != 0;
    Acc<C> c;
    // gbar and Vbar
    fill<C>(X, V, nl, n, nl);
    prod<C, false, false>(c, lx, X, kd, L);  // X V          (n x nl)
    store_rows<C>(T1, c, L);
    fill<C>(X, T1);
    prod<C, true, false>(c, lv, X, kd, L);  // V^H X V      (nl x nl)
    store_rows<C>(Lam, c, L);
    fill<C>(X, xs, n, n, n);
    prod<C, true, false>(c, lv, X, kd, L);  // V^H X        (nl x n)
    store_rows<C>(T2, c, L);
    fill<C>(X, g, nl, nl, nl);
    prod<C, false, false>(c, ws_left<C>(T1), X, kl, L);  // X V g        (n x nl)
    store_rows<C>(Bp, c, L);
    fill<C>(X, T2);
    prod<C, false, false>(c, lg, X, kl, L);  // g V^H X      (nl x n)
    {
      double2* gv = sa.grad_v + (own ? (long long)p * nl * n : k * (sa.v_ks ? (long long)nl * n : 0));
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        if (r < nl && cc < n)
          grad_put(gv + (long long)r * n + cc, cadd(c.get(0, j, q), cconj(Bp[cc * NP + r])), own);
      });
    }
    // B = P = g H01, A = Q = H10 g
    fill<C>(X, h01, nl, nl, nl);
    prod<C, false, false>(c, lg, X, kl, L);
    store_rows<C>(Bp, c, L);
    fill<C>(X, g, nl, nl, nl);
    if (h10) prod<C, false, false>(c, lh10, X, kl, L);
    else prod<C, true, false>(c, lh01, X, kl, L);
    store_rows<C>(Aq, c, L);
    // Smith doubling for Lam - Q Lam P = gbar
    int status = kOk, it = 0;
    for (;;) {
      ++it;
      double m = 0.0;
      int bad = 0;
      auto measure = [&]() {
        smem::each<C>(L, [&](int, int j, int q, int, int) {
          const double2 v = c.get(0, j, q);
          bad |= !cfinite(v);
          m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
        });
      };
      fill<C>(X, Lam);
      prod<C, false, false>(c, ws_left<C>(Aq), X, kl, L);
      store_rows<C>(Tt, c, L);
      fill<C>(X, Bp);
      prod<C, false, false>(c, ws_left<C>(Tt), X, kl, L);
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        double2& e = Lam[r * NP + cc];
        const double2 v = cadd(e, c.get(0, j, q));
        e = v;
        bad |= !cfinite(v);
      });
      prod<C, false, false>(c, ws_left<C>(Bp), X, kl, L);
      measure();
      store_rows<C>(Bp, c, L);  // own rows; the others' are in X
      fill<C>(X, Aq);
      prod<C, false, false>(c, ws_left<C>(Aq), X, kl, L);
      measure();
      store_rows<C>(Aq, c, L);
      if (block_any(bad)) {
        status = kNonFinite;
        break;
      }
      m = block_max(m, sh.red);
      if (m < sa.tol) break;
      if (it >= sa.maxiter) {
        status = kMaxIter;
        break;
      }
    }
    if (status == kOk) {
      const long long slot = own ? (long long)p : k;
      double2* g00 = sa.grad_h00 + slot * nl * nl;
      double2* g01 = sa.grad_h01 + slot * nl * nl;
      double2* g10 = sa.grad_h10 ? sa.grad_h10 + slot * nl * nl : nullptr;
      fill<C>(X, g, nl, nl, nl);
      prod<C, false, false>(c, lh01, X, kl, L);  // H01 g
      store_rows<C>(U, c, L);
      prod<C, false, false>(c, ws_left<C>(Lam), X, kl, L);  // Lam g
      fill<C>(X, c, L);
      prod<C, false, false>(c, lg, X, kl, L);  // H00bar = g Lam g
      store_rows<C>(T1, c, L);
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        if (r < nl && cc < nl) grad_put(g00 + r * nl + cc, c.get(0, j, q), own);
      });
      fill<C>(X, U);
      prod<C, false, false>(c, ws_left<C>(T1), X, kl, L);  // H10bar = H00bar H01 g
      store_rows<C>(Tt, c, L);
      if (h10) fill<C>(X, h10, nl, nl, nl);
      else fill<C>(X, h01, nl, nl, nl);
      if (h10) prod<C, false, false>(c, lg, X, kl, L);  // g H10
      else prod<C, false, true>(c, lg, X, kl, L);
      store_rows<C>(T2, c, L);
      fill<C>(X, T1);
      prod<C, false, false>(c, ws_left<C>(T2), X, kl, L);  // H01bar = g H10 H00bar
      tiles<C>(L, [&](int j, int q, int r, int cc) {
        if (r < nl && cc < nl) {
          if (h10) {
            grad_put(g01 + r * nl + cc, c.get(0, j, q), own);
            if (g10) grad_put(g10 + r * nl + cc, Tt[r * NP + cc], own);
          } else {
            grad_put(g01 + r * nl + cc, cadd(c.get(0, j, q), cconj(Tt[cc * NP + r])), own);
          }
        }
      });
    }
    __syncthreads();
    if (tid == 0) {
      if (sa.status_out) sa.status_out[p] = status;
      if (sa.iters_out) sa.iters_out[p] = it;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ full device G --
// Every block of G = A^-1 for one point (negfpy core/negf.py:253-303 builds it
// densely with SuperLU), in two kernels.  The first, one block per point: a left
// sweep keeps g^L_i, W_i = g^L_i C_i and V_i = C_i^H g^L_i, and the diagonal
// follows backwards without further inverses,
//   G_{L-1,L-1} = g^L_{L-1},  G_ii = g^L_i + W_i G_{i+1,i+1} V_i.
// The second walks each column up and each row left from its diagonal block,
//   G_ij = W_i G_{i+1,j},  G_ji = G_{j,i+1} V_i   (i < j),
// one block per point, column and direction: these 2 (L - 1) walks are
// independent, and on one block their L (L - 1) products were most of the time.
// Workspace per point: U and L slots each of G_ii, W_i, V_i, then Sigma_L, Sigma_R.
template <class C>
constexpr size_t full_ws(int n, int L) { return (1 + 3 * (size_t)L) * C::MAT + 2 * (size_t)n * n; }

// The thread's elements -> block (bi, bj) of G.
template <class C>
__device__ __forceinline__ void put_block(double2* Gp, long long dim, int bi, int bj, const Acc<C>& c, int n,
                                          const Lane& L) {
  smem::each<C>(L, [&](int, int j, int q, int r, int cc) {
    if (r < n && cc < n) Gp[((long long)bi * n + r) * dim + (long long)bj * n + cc] = c.get(0, j, q);
  });
}

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) full_diag_kernel(FullArgs fa, int first, double2* ws) {
  constexpr int MAT = C::MAT, NP = C::NP;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  const RgfArgs& a = fa.r;
  const int n = a.n, nlay = a.L, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  const long long dim = (long long)nlay * n;
  double2* const U = ws + (long long)blockIdx.x * full_ws<C>(n, nlay);
  double2 *const gl = U + MAT, *const Ws = gl + (long long)nlay * MAT, *const Vs = Ws + (long long)nlay * MAT;
  double2 *const sigL = Vs + (long long)nlay * MAT, *const sigR = sigL + (long long)n * n;
  const int p = first + blockIdx.x;
  const int lst = a.lead_status ? a.lead_status[p] : 0;
  if (lst != kOk) {
    if (tid == 0 && a.status_out) a.status_out[p] = lst;
    return;
  }
  const long long k = a.kidx ? (long long)a.kidx[p] : 0;
  const double2 z = z_of(a.omega[p], a.eta_dev[p]);
  const double2* D = a.D + k * a.d_ks;
  const double2* Cg = a.C + k * a.c_ks;
  self_energy<C>(sigL, a.VL + k * a.vl_ks, a.gL + (long long)p * a.gl_ps, n, a.nl, U, X, L);
  self_energy<C>(sigR, a.VR + k * a.vr_ks, a.gR + (long long)p * a.gr_ps, n, a.nr, U, X, L);
  for (int e = tid; e < n * n; e += C::NTH) {
    fa.sigL_out[(long long)p * n * n + e] = sigL[e];
    fa.sigR_out[(long long)p * n * n + e] = sigR[e];
  }
  Acc<C> c;
  int status = kOk;
  for (int l = 0; l < nlay; ++l) {
    if (l == 0) {
      load_tiles<C>(c, sigL, n, L);
    } else {
      const Left Cl{Cg + (long long)(l - 1) * a.c_ls, n, n, n};
      // X holds g_{l-1}
      prod<C, true, false>(c, Cl, X, kch, L);  // V = C^H g
      store_rows<C>(Vs + (l - 1) * MAT, c, L);
      fill<C>(X, Cl.p, n, n, n);
      prod<C, false, false>(c, ws_left<C>(gl + (l - 1) * MAT), X, kch, L);  // W = g C
      store_rows<C>(Ws + (l - 1) * MAT, c, L);
      fill<C>(X, c, L);
      prod<C, true, false>(c, Cl, X, kch, L);  // C^H W
    }
    minus_d<C>(c, D + (long long)l * a.d_ls, l == nlay - 1 ? sigR : nullptr, z, n, L);
    status = invert_to<C>(gl + l * MAT, c, n, X, sh.gj, L);
    if (status != kOk) break;
  }
  if (status == kOk) {
    double2* Gp = fa.G + (long long)p * dim * dim;
    // diagonal, backwards: G_ii = g^L_i + W_i G_{i+1,i+1} V_i (into the g^L slot)
    for (int i = nlay - 1; i >= 0; --i) {
      if (i < nlay - 1) {
        fill<C>(X, gl + (i + 1) * MAT);
        prod<C, false, false>(c, ws_left<C>(Ws + i * MAT), X, kch, L);
        store_rows<C>(U, c, L);
        fill<C>(X, Vs + i * MAT);
        prod<C, false, false>(c, ws_left<C>(U), X, kch, L);
        tiles<C>(L, [&](int j, int q, int r, int cc) { c.set(0, j, q, cadd(gl[i * MAT + r * NP + cc], c.get(0, j, q))); });
        store_rows<C>(gl + i * MAT, c, L);
      } else {
        tiles<C>(L, [&](int j, int q, int r, int cc) { c.set(0, j, q, gl[i * MAT + r * NP + cc]); });
      }
      put_block<C>(Gp, dim, i, i, c, n, L);
    }
  }
  if (tid == 0 && a.status_out) a.status_out[p] = status;
  if (tid == 0) reinterpret_cast<int*>(U)[0] = status;  // for the walks
}

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) full_walk_kernel(FullArgs fa, int first, const double2* ws) {
  constexpr int MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  const RgfArgs& a = fa.r;
  const int n = a.n, nlay = a.L, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  const long long dim = (long long)nlay * n;
  const int walks = 2 * (nlay - 1), s = blockIdx.x / walks, w = blockIdx.x % walks;
  const int j = nlay - 1 - w / 2;  // longest walks first
  const double2* const U = ws + (long long)s * full_ws<C>(n, nlay);
  const double2 *const gl = U + MAT, *const Ws = gl + (long long)nlay * MAT, *const Vs = Ws + (long long)nlay * MAT;
  const int p = first + s;
  if ((a.lead_status && a.lead_status[p] != kOk) || reinterpret_cast<const int*>(U)[0] != kOk) return;
  double2* Gp = fa.G + (long long)p * dim * dim;
  Acc<C> c;
  if (w & 1) {
    for (int i = j - 1; i >= 0; --i) {  // G_ji = G_{j,i+1} V_i; the left operand is the warp's own rows of G
      fill<C>(X, Vs + i * MAT);
      const Left g = i == j - 1 ? ws_left<C>(gl + j * MAT)
                                : Left{Gp + (long long)j * n * dim + (long long)(i + 1) * n, (int)dim, n, n};
      prod<C, false, false>(c, g, X, kch, L);
      put_block<C>(Gp, dim, j, i, c, n, L);
      __syncwarp();
    }
  } else {
    fill<C>(X, gl + j * MAT);
    for (int i = j - 1; i >= 0; --i) {  // G_ij = W_i G_{i+1,j}
      prod<C, false, false>(c, ws_left<C>(Ws + i * MAT), X, kch, L);
      put_block<C>(Gp, dim, i, j, c, n, L);
      if (i > 0) fill<C>(X, c, L);
    }
  }
}

}  // namespace mid
}  // namespace negf
