// The FP32 sweeps of the mixed and the refined device solve for orders up to 96,
// one (omega, k) point per thread block, on the layout of negf_mid.cuh: the
// right operand of a product in shared memory, its result and the matrix being
// inverted in registers, the left operand read from global memory (L2) straight
// into MMA fragments.  Before, both operands of every 16 x 16 tile came from
// L2/L1, C was converted and padded into the workspace for each product, and an
// FP32 inverse streamed two buffers through L2 per update.
//
// Arithmetic as in negf_mixed.cuh, operation for operation: 3 x TF32 products on
// mma.sync m16n8k8 with every chunk's passes started from zero and added with a
// rounded FP32 add, the division-free FP32 Gauss-Jordan, FP64 self-energies,
// residuals and trace; results are bitwise those of the workspace kernels.
//
// Measured, 592 points, 8 layers, before and after, ms: refined n = 24 1.33 -> 0.89,
// 48 5.46 -> 3.45, 63 9.1 -> 6.1, 96 25.8 -> 18.6; mixed 0.48 -> 0.32, 1.51 -> 1.10,
// 2.7 -> 1.8, 7.2 -> 5.9.  Bound by the FP64 pipe in the residuals (27 % of the time at
// n = 48), the tensor pipe in the FP32 products (20 %) and the pivot steps, in turn.
//
// FP64 parts use warp w for rows 8 w .. 8 w + 7 (negf_mid.cuh); FP32 parts use
// warp w for rows 16 (w / 2) .. + 15 and one half of the columns.
#pragma once
#include "negf_mid.cuh"
#include "negf_mixed.cuh"

namespace negf {
namespace mid {

using mixed::fmulc;
using mixed::to_f;

template <class C>
struct Lane32 {
  int g, t, R, c0;  // lane's group and member, first row, first own column
  __device__ __forceinline__ Lane32() {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    g = l >> 2;
    t = l & 3;
    R = (w >> 1) * 16;
    c0 = (w & 1) * (C::NP / 2) + 2 * t;
  }
  __device__ __forceinline__ int row(int q) const { return R + g + 8 * (q >> 1); }
  __device__ __forceinline__ int col(int j, int q) const { return c0 + 8 * j + (q & 1); }
};
// The thread's elements of an FP32 matrix: element (j, q) at (row(q), col(j, q)).
template <class C>
struct Acc32 {
  static constexpr int TN = C::NP / 16;  // 16 x 8 tiles of the warp
  float re[TN][4], im[TN][4];
  __device__ __forceinline__ float2 get(int j, int q) const { return make_float2(re[j][q], im[j][q]); }
  __device__ __forceinline__ void set(int j, int q, float2 v) {
    re[j][q] = v.x;
    im[j][q] = v.y;
  }
};
template <class C, class F>
__device__ __forceinline__ void each32(const Lane32<C>& L, F&& f) {
#pragma unroll
  for (int j = 0; j < Acc32<C>::TN; ++j) {
    if (j % 3 == 0) asm volatile("" ::: "memory");  // loads of three tiles in flight
#pragma unroll
    for (int q = 0; q < 4; ++q) f(j, q, L.row(q), L.col(j, q));
  }
}
// Shared FP32 matrix: row stride NP, the column XORed by 4 (row mod 4): the 4 x 4
// blocks that a half warp reads as B fragments fall into 16 different banks.
template <int NP>
__device__ __forceinline__ int sidx32(int r, int c) { return r * NP + (c ^ ((r & 3) << 2)); }

// X <- an n x n FP64 matrix rounded, zeros outside / the thread's elements.
template <class C>
__device__ __forceinline__ void fill32(float2* X, const double2* __restrict__ src, int n) {
  __syncthreads();
#pragma unroll 4
  for (int idx = threadIdx.x; idx < C::MAT; idx += C::NTH) {
    const int r = idx / C::NP, c = idx - r * C::NP;
    X[sidx32<C::NP>(r, c)] = (r < n && c < n) ? to_f(src[(long long)r * n + c]) : make_float2(0.f, 0.f);
  }
  __syncthreads();
}
template <class C>
__device__ __forceinline__ void fill32(float2* X, const Acc32<C>& c, const Lane32<C>& L) {
  __syncthreads();
  each32<C>(L, [&](int j, int q, int r, int cc) { X[sidx32<C::NP>(r, cc)] = c.get(j, q); });
  __syncthreads();
}
template <class C>
__device__ __forceinline__ void store32(float2* G, const Acc32<C>& c, const Lane32<C>& L) {
  each32<C>(L, [&](int j, int q, int r, int cc) { G[r * C::NP + cc] = c.get(j, q); });
}

// Left operands: a padded FP32 workspace matrix, or an n x n FP64 matrix rounded.
struct Left32 {
  const float2* p;
  int ld;
  __device__ __forceinline__ float2 get(int r, int k) const { return p[r * ld + k]; }
};
struct LeftC {
  const double2* p;
  int n;
  __device__ __forceinline__ float2 get(int r, int k) const {
    return (r < n && k < n) ? to_f(p[(long long)r * n + k]) : make_float2(0.f, 0.f);
  }
};

// c = op(A) X on 3 x TF32 (op: conjugate transpose with AC), kch chunks of 8; the
// next chunk's A is loaded under the current chunk's MMAs.
template <class C, bool AC, class A>
__device__ __forceinline__ void prod32(Acc32<C>& c, const A& a, const float2* X, int kch, const Lane32<C>& L) {
  constexpr int NP = C::NP, TN = Acc32<C>::TN;
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) c.re[j][q] = c.im[j][q] = 0.f;
  auto load = [&](float2(&v)[4], int kc) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = L.R + L.g + 8 * (q & 1), k = kc * 8 + L.t + 4 * (q >> 1);
      v[q] = AC ? a.get(k, r) : a.get(r, k);
      if (AC) v[q].y = -v[q].y;
    }
  };
  const int n0 = L.c0 - 2 * L.t + L.g;  // column of the B fragments
  float2 av[4], an[4];
  load(av, 0);
#pragma unroll 1
  for (int kc = 0; kc < kch; ++kc) {
    load(an, kc + 1 < kch ? kc + 1 : 0);
    mixed::AFrag f;
#pragma unroll
    for (int q = 0; q < 4; ++q) mixed::set_a(f, q, av[q]);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      mixed::BFrag b;
#pragma unroll
      for (int q = 0; q < 2; ++q) mixed::set_b(b, q, X[sidx32<NP>(kc * 8 + L.t + 4 * q, n0 + 8 * j)]);
      float pr[4] = {0.f, 0.f, 0.f, 0.f}, pi[4] = {0.f, 0.f, 0.f, 0.f};
      mixed::cmma3(pr, pi, f, b);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c.re[j][q] = __fadd_rn(c.re[j][q], pr[q]);
        c.im[j][q] = __fadd_rn(c.im[j][q], pi[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) av[q] = an[q];
  }
}

// ------------------------------------------------------- FP32 Gauss-Jordan --
// smem::gj_invert in FP32 (see there for the algorithm; pivot keys as in
// mixed::gj_invert32): the inverse of the matrix in m into the shared matrix X,
// which is also the scratch.  Ends with the block synchronised.
template <class C>
struct GJ32 {
  alignas(16) float2 lam[2];
  unsigned key[8][C::NW];
  int fail;
  int newpos[C::NP];
  int cmapinv[C::NP];
};
template <class C>
__device__ __forceinline__ int gj_invert32(Acc32<C>& m, float2* X, int n, const Lane32<C>& L, GJ32<C>& sh) {
  constexpr int NP = C::NP, NW = C::NW, LPR = C::LPR, EPT = C::EPT, PS = C::PS, PE = C::PE, TN = Acc32<C>::TN;
  static_assert(2 * PE + 8 * NP <= 2 * C::BUF, "panel scratch");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool work = NW == C::WW || warp < C::WW;
  const bool live = C::NTH == NP * LPR || tid < NP * LPR;
  const int pr_own = live ? tid / LPR : 0, cl = tid % LPR, prow = pr_own * PS;
  float2* const Bp = X + 2 * PE;
  int pos[2] = {L.R + L.g, L.R + L.g + 8};
  const bool bk = warp == NW - 1;
  constexpr bool kAll = NW <= C::WW + 1;
  constexpr int RL = (NP + 31) / 32;
  int cm[RL];
#pragma unroll
  for (int i = 0; i < RL; ++i) cm[i] = lane + 32 * i;

  __syncthreads();
#pragma unroll 1
  for (int k0 = 0, par = 0; k0 < n; k0 += 8, par ^= 1) {
    const int jmax = (n - k0) < 8 ? (n - k0) : 8;
    float2* const P0 = X + par * PE;
    float2* const P1 = X + (par ^ 1) * PE;
    const int pj = (k0 - (L.c0 - 2 * L.t)) >> 3;  // the panel's tile among the warp's, if in range
    unsigned key0 = 0u;
#pragma unroll
    for (int j = 0; j < TN; ++j)
      if (j == pj) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float2* row = P0 + pos[i] * PS + 2 * L.t;
          row[0] = m.get(j, 2 * i);
          row[1] = m.get(j, 2 * i + 1);
          if (L.t == 0 && pos[i] >= k0 && pos[i] < n) key0 = max(key0, mixed::pivot_key32(m.get(j, 2 * i), pos[i]));
        }
      }
    key0 = __reduce_max_sync(0xffffffffu, key0);
    if (lane == 0) sh.key[0][warp] = key0;
    if (tid == 0) sh.lam[0] = make_float2(1.f, 0.f);
    __syncthreads();
    if (work || bk) {
      float2 av[EPT];
#pragma unroll
      for (int q = 0; q < EPT; ++q) av[q] = P0[prow + cl + LPR * q];
      bool cand = live && pr_own >= k0 && pr_own < n;
      int fail = kOk;
      int lg[RL];
#pragma unroll
      for (int i = 0; i < RL; ++i) lg[i] = lane + 32 * i;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= jmax) break;
        const float2* Pc = (j & 1) ? P1 : P0;
        float2* Pn = (j & 1) ? P0 : P1;
        const float2 fv = Pc[prow + j];
        const float2 lam = sh.lam[j & 1];
        const unsigned key =
            __reduce_max_sync(0xffffffffu, lane < (j == 0 || kAll ? NW : C::WW) ? sh.key[j][lane] : 0u);
        const bool stop = key - 256u >= 0x7f800000u - 256u;
        const int pr = min((int)(255u - (key & 255u)), NP - 1);
        const int ex = (int)(key >> 23);
        const float sc = (ex != 0 && ex < 254) ? __uint_as_float((unsigned)(254 - ex) << 23) : 1.0f;
        const float2* prow_p = Pc + pr * PS;
        const float2 piv = prow_p[j];
        const float2 ps = make_float2(piv.x * sc, piv.y * sc);
        unsigned nk = 0u;
        if (work) {
          float2 mv[EPT];
#pragma unroll
          for (int q = 0; q < EPT; ++q) mv[q] = prow_p[cl + LPR * q];
          const bool isp = pr_own == pr;
          cand = cand && !isp;
          const float2 bb = isp ? lam : fv;
          const float nsc = isp ? sc : -sc;
          const float2 nb = make_float2(bb.x * nsc, bb.y * nsc);
          const float2 pe = isp ? make_float2(0.f, 0.f) : ps;
#pragma unroll
          for (int qq = 0; qq < EPT; ++qq) {
            const int q = (qq + (j + 1) / LPR) % EPT;
            const int c = cl + LPR * q;
            const bool pivcol = q == j / LPR && cl == j % LPR;
            const float2 mq = pivcol ? lam : mv[q];
            float2 v = make_float2(fmaf(nb.x, mq.x, -nb.y * mq.y), fmaf(nb.x, mq.y, nb.y * mq.x));
            cfma(v, pivcol ? make_float2(0.f, 0.f) : pe, av[q]);
            if (live) Pn[prow + c] = v;
            av[q] = v;
            if (j + 1 < 8 && qq == 0) {
              if (cl == (j + 1) % LPR && cand) nk = mixed::pivot_key32(v, pr_own);
              nk = __reduce_max_sync(0xffffffffu, nk);
            }
          }
        }
        if (j + 1 < 8 && lane == 0) sh.key[j + 1][warp] = nk;
        if (bk) {
          const float2 ln = fmulc(lam, ps);
          if (lane == 0) sh.lam[(j + 1) & 1] = ln;
          const int k = k0 + j;
          int x = lg[0];
#pragma unroll
          for (int i = 1; i < RL; ++i) x = (pr >> 5) == i ? lg[i] : x;
          const int bl = __shfl_sync(0xffffffffu, x, pr & 31);
#pragma unroll
          for (int i = 0; i < RL; ++i) {
            lg[i] = lane + 32 * i == pr ? k : (lg[i] == k ? bl : lg[i]);
            cm[i] = cm[i] == k ? bl : (cm[i] == bl ? k : cm[i]);
            if (j + 1 == jmax && lane + 32 * i < NP) sh.newpos[lane + 32 * i] = lg[i];
          }
        }
        if (stop) fail = fail ? fail : (key <= 255u ? kSingular : kNonFinite);
        if (j + 1 < jmax) {
          if (kAll) __syncthreads();
          else asm volatile("bar.sync 1, %0;" ::"n"(32 * (C::WW + 1)) : "memory");
        }
      }
      if (bk && lane == 0) sh.fail = fail;
    }
    __syncthreads();
    if (sh.fail) return sh.fail;
    int np[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      np[i] = sh.newpos[pos[i]];
      if ((unsigned)(np[i] - k0) < (unsigned)jmax) {
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            Bp[sidx32<NP>(np[i] - k0, L.c0 + 8 * j + q)] = m.get(j, 2 * i + q);
            m.set(j, 2 * i + q, make_float2(0.f, 0.f));
          }
      }
    }
    const float2* P = (jmax & 1) ? P1 : P0;
    const float2 il = mixed::crecip_smith32(sh.lam[jmax & 1]);
    mixed::AFrag a;
#pragma unroll
    for (int q = 0; q < 4; ++q) mixed::set_a(a, q, fmulc(P[pos[q & 1] * PS + L.t + 4 * (q >> 1)], il));
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      if (j == pj) {
#pragma unroll
        for (int q = 0; q < 4; ++q) m.set(j, q, fmulc(P[pos[q >> 1] * PS + 2 * L.t + (q & 1)], il));
      } else {
        mixed::BFrag b;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int kk = L.t + 4 * q;
          const float2 v = Bp[sidx32<NP>(kk, L.c0 - 2 * L.t + 8 * j + L.g)];
          mixed::set_b(b, q, kk < jmax ? v : make_float2(0.f, 0.f));
        }
        float pr[4] = {0.f, 0.f, 0.f, 0.f}, pi[4] = {0.f, 0.f, 0.f, 0.f};
        mixed::cmma3(pr, pi, a, b);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          m.re[j][q] = __fadd_rn(m.re[j][q], pr[q]);
          m.im[j][q] = __fadd_rn(m.im[j][q], pi[q]);
        }
      }
    }
    pos[0] = np[0];
    pos[1] = np[1];
  }
  if (bk)
#pragma unroll
    for (int i = 0; i < RL; ++i)
      if (lane + 32 * i < NP) sh.cmapinv[cm[i]] = lane + 32 * i;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = sh.cmapinv[L.c0 + 8 * j + q];
#pragma unroll
      for (int i = 0; i < 2; ++i) X[sidx32<NP>(pos[i], c)] = m.get(j, 2 * i + q);
    }
  __syncthreads();
  return kOk;
}
// X (swizzled) -> row-major workspace.
template <class C>
__device__ __forceinline__ void copy_x32(float2* G, const float2* X) {
  for (int idx = threadIdx.x; idx < C::MAT; idx += C::NTH) {
    const int r = idx / C::NP, c = idx - r * C::NP;
    G[idx] = X[sidx32<C::NP>(r, c)];
  }
}

// c = z - D [- S1] [- S2] - c, the FP64 terms combined before the rounding;
// identity in the padding.
template <class C>
__device__ __forceinline__ void minus_d32(Acc32<C>& c, bool have, const double2* D, const double2* S1, const double2* S2,
                                          double2 z, int n, const Lane32<C>& L) {
  each32<C>(L, [&](int j, int q, int r, int cc) {
    if (r < n && cc < n) {
      double2 w = cneg(D[r * n + cc]);
      if (S1) w = csub(w, S1[r * n + cc]);
      if (S2) w = csub(w, S2[r * n + cc]);
      if (r == cc) w = cadd(w, z);
      const float2 x = have ? c.get(j, q) : make_float2(0.f, 0.f);
      c.set(j, q, make_float2((float)(w.x - (double)x.x), (float)(w.y - (double)x.y)));
    } else {
      c.set(j, q, make_float2(r == cc ? 1.f : 0.f, 0.f));
    }
  });
}

template <class C>
struct Shared32 {
  GJ32<C> gj;
  double red[40];
  int point;
};
template <class C>
constexpr size_t shared32_bytes() { return (size_t)C::BUF * 16 + sizeof(Shared32<C>); }

// ------------------------------------------------------------- mixed solve --
// Sigma, Gamma and trace in FP64, the RGF sweep in FP32.  Workspace: three FP64
// matrices, Sigma_L, Sigma_R, three FP32 matrices (g, G_0, U).
template <class C>
constexpr size_t mixed_ws_bytes(int n) { return (3 * (size_t)C::MAT + 2 * (size_t)n * n) * 16 + 3 * (size_t)C::MAT * 8; }

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) mixed_kernel(RgfArgs a, unsigned char* ws) {
  constexpr int NP = C::NP, MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  float2* const X32 = reinterpret_cast<float2*>(smraw);
  Shared32<C>& sh = *reinterpret_cast<Shared32<C>*>(X + C::BUF);
  const int n = a.n, nlay = a.L, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  const Lane32<C> M;
  unsigned char* blk = ws + (long long)blockIdx.x * mixed_ws_bytes<C>(n);
  double2 *const U64 = reinterpret_cast<double2*>(blk), *const G64 = U64 + MAT, *const GL = G64 + MAT;
  double2 *const sigL = GL + MAT, *const sigR = sigL + (long long)n * n;
  float2 *const gs = reinterpret_cast<float2*>(sigR + (long long)n * n), *const G0 = gs + MAT, *const U = G0 + MAT;

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
    self_energy<C>(sigL, a.VL + k * a.vl_ks, a.gL + (long long)p * a.gl_ps, n, a.nl, U64, X, L);
    self_energy<C>(sigR, a.VR + k * a.vr_ks, a.gR + (long long)p * a.gr_ps, n, a.nr, U64, X, L);
    Acc32<C> c;
    int status = kOk;
    for (int l = 0; l < nlay; ++l) {
      if (l > 0) {
        const LeftC Cl{Cg + (long long)(l - 1) * a.c_ls, n};
        fill32<C>(X32, Cl.p, n);
        prod32<C, false>(c, Left32{G0, NP}, X32, kch, M);  // U = G_{0,l-1} C
        store32<C>(U, c, M);
        prod32<C, false>(c, Left32{gs, NP}, X32, kch, M);  // W = g_{l-1} C
        fill32<C>(X32, c, M);
        prod32<C, true>(c, Cl, X32, kch, M);  // C^H W
      }
      minus_d32<C>(c, l > 0, D + (long long)l * a.d_ls, l == 0 ? sigL : nullptr, l == nlay - 1 ? sigR : nullptr, z, n, M);
      status = gj_invert32<C>(c, X32, n, M, sh.gj);
      if (status != kOk) break;
      if (l + 1 < nlay) copy_x32<C>(gs, X32);
      if (l == 0) {
        copy_x32<C>(G0, X32);
      } else {
        prod32<C, false>(c, Left32{U, NP}, X32, kch, M);  // G_{0,l} = U g_l
        store32<C>(G0, c, M);
      }
      __syncthreads();
    }
    double tval = 0.0;
    if (status == kOk) {
      for (int e = tid; e < MAT; e += C::NTH) {
        const float2 v = G0[e];
        G64[e] = make_double2((double)v.x, (double)v.y);
      }
      __syncthreads();
      tval = trace_t<C>(sigL, sigR, G64, GL, U64, n, max(n, max(a.nl, a.nr)), X, sh.red, L);
      if (!isfinite(tval)) status = kNonFinite;
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------- refined solve --
// FP32 block LU factors, FP64 iterative refinement of the right-contact column
// of A X = E_R (the steps and the stopping rule are described in
// negf_refine.cu).  Workspace: two FP64 matrices, L slots of X, Sigma_L,
// Sigma_R, 2 L + 1 FP32 matrices (g_l, y_l / d_l, C^H y).
template <class C>
constexpr size_t refine_ws_bytes(int n, int L) {
  return ((2 + (size_t)L) * C::MAT + 2 * (size_t)n * n) * 16 + (2 * (size_t)L + 1) * C::MAT * 8;
}

template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC)
refine_kernel(RgfArgs a, unsigned char* ws, double tol, int maxit, int* steps_out) {
  constexpr int NP = C::NP, MAT = C::MAT;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const X = reinterpret_cast<double2*>(smraw);
  float2* const X32 = reinterpret_cast<float2*>(smraw);
  Shared32<C>& sh = *reinterpret_cast<Shared32<C>*>(X + C::BUF);
  const int n = a.n, nlay = a.L, tid = threadIdx.x, kch = (n + 7) >> 3;
  const Lane L = smem::lane_geo<C>();
  const Lane32<C> M;
  unsigned char* blk = ws + (long long)blockIdx.x * refine_ws_bytes<C>(n, nlay);
  double2 *const U64 = reinterpret_cast<double2*>(blk), *const GL = U64 + MAT;
  double2* const X64 = GL + MAT;
  double2 *const sigL = X64 + (long long)nlay * MAT, *const sigR = sigL + (long long)n * n;
  float2* const gs = reinterpret_cast<float2*>(sigR + (long long)n * n);
  float2 *const ys = gs + (long long)nlay * MAT, *const cy = ys + (long long)nlay * MAT;

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
        if (steps_out) steps_out[p] = 0;
      }
      continue;
    }
    const long long k = a.kidx ? (long long)a.kidx[p] : 0;
    const double2 z = z_of(a.omega[p], a.eta_dev[p]);
    const double2* D = a.D + k * a.d_ks;
    const double2* Cg = a.C + k * a.c_ks;
    auto Cl = [&](int l) { return Cg + (long long)l * a.c_ls; };
    self_energy<C>(sigL, a.VL + k * a.vl_ks, a.gL + (long long)p * a.gl_ps, n, a.nl, U64, X, L);
    self_energy<C>(sigR, a.VR + k * a.vr_ks, a.gR + (long long)p * a.gr_ps, n, a.nr, U64, X, L);
    Acc32<C> c;
    int status = kOk, steps = 0;
    // 1. FP32 left sweep; g_l kept in slot l.
    for (int l = 0; l < nlay; ++l) {
      if (l > 0) {
        fill32<C>(X32, Cl(l - 1), n);
        prod32<C, false>(c, Left32{gs + (l - 1) * MAT, NP}, X32, kch, M);  // g_{l-1} C_{l-1}
        fill32<C>(X32, c, M);
        prod32<C, true>(c, LeftC{Cl(l - 1), n}, X32, kch, M);  // C^H g C
      }
      minus_d32<C>(c, l > 0, D + (long long)l * a.d_ls, l == 0 ? sigL : nullptr, l == nlay - 1 ? sigR : nullptr, z, n, M);
      status = gj_invert32<C>(c, X32, n, M, sh.gj);
      if (status != kOk) break;
      copy_x32<C>(gs + l * MAT, X32);
    }
    double tval = 0.0;
    if (status == kOk) {
      // 2. Last block column in FP32, widened into X64.
      auto widen = [&](int i, int r, int cc, float2 v) {
        X64[(long long)i * MAT + r * NP + cc] =
            (r < n && cc < n) ? make_double2((double)v.x, (double)v.y) : make_double2(0.0, 0.0);
      };
      for (int idx = tid; idx < MAT; idx += C::NTH) {  // X_{L-1} = g_{L-1}, still in X32
        const int r = idx / NP, cc = idx - r * NP;
        widen(nlay - 1, r, cc, X32[sidx32<NP>(r, cc)]);
      }
      for (int i = nlay - 2; i >= 0; --i) {
        prod32<C, false>(c, LeftC{Cl(i), n}, X32, kch, M);  // C_i X_{i+1}
        fill32<C>(X32, c, M);
        prod32<C, false>(c, Left32{gs + i * MAT, NP}, X32, kch, M);  // X_i = g_i C_i X_{i+1}
        fill32<C>(X32, c, M);
        each32<C>(M, [&](int j, int q, int r, int cc) { widen(i, r, cc, c.get(j, q)); });
      }
      // 3. Refinement.
      double nu_prev = 0.0;
      bool done = false;
      for (int it = 1; it <= maxit && !done && status == kOk; ++it) {
        steps = it;
        // forward: R_i in FP64, t_i = R_i + C_{i-1}^H y_{i-1}, y_i = g_i t_i
        for (int i = 0; i < nlay; ++i) {
          const double2* Xi = X64 + (long long)i * MAT;
          if (i > 0) {
            fill32<C>(X32, c, M);  // y_{i-1}
            prod32<C, true>(c, LeftC{Cl(i - 1), n}, X32, kch, M);
            store32<C>(cy, c, M);
          }
          // D_i X_i + C_{i-1}^H X_{i-1} + C_i X_{i+1} + Sigma X_i at the ends
          Acc<C> r64;
          auto term = [&](const double2* B, const double2* A, bool ct, bool first) {
            __syncthreads();
            load_x<C>(X, B, NP, NP, NP);
            __syncthreads();
            const Left l{A, n, n, n};
            if (first) prod<C, false, false>(r64, l, X, kch, L);
            else if (ct) prod<C, true, false, true>(r64, l, X, kch, L);
            else prod<C, false, false, true>(r64, l, X, kch, L);
          };
          term(Xi, D + (long long)i * a.d_ls, false, true);
          if (i > 0) term(Xi - MAT, Cl(i - 1), true, false);
          if (i < nlay - 1) term(Xi + MAT, Cl(i), false, false);
          if (i == 0) term(Xi, sigL, false, false);
          if (i == nlay - 1) term(Xi, sigR, false, false);
          __syncthreads();
          tiles<C>(L, [&](int j, int q, int r, int cc) {
            float2 v = make_float2(0.f, 0.f);
            if (r < n && cc < n) {
              // R = E - (z X - D X - C^H X - C X - Sigma X)
              double2 rv = csub(r64.get(0, j, q), cmul(z, Xi[r * NP + cc]));
              if (i == nlay - 1 && r == cc) rv.x += 1.0;
              const float2 y = i > 0 ? cy[r * NP + cc] : make_float2(0.f, 0.f);
              v = make_float2((float)rv.x + y.x, (float)rv.y + y.y);
            }
            X32[sidx32<NP>(r, cc)] = v;
          });
          __syncthreads();
          prod32<C, false>(c, Left32{gs + i * MAT, NP}, X32, kch, M);  // y_i
          store32<C>(ys + i * MAT, c, M);
        }
        // backward: d_{L-1} = y_{L-1}, d_i = y_i + g_i C_i d_{i+1}; X += d
        double dmax = 0.0, xmax = 0.0;
        for (int i = nlay - 1; i >= 0; --i) {
          if (i < nlay - 1) {
            fill32<C>(X32, c, M);                               // d_{i+1}
            prod32<C, false>(c, LeftC{Cl(i), n}, X32, kch, M);  // C_i d_{i+1}
            fill32<C>(X32, c, M);
            prod32<C, false>(c, Left32{gs + i * MAT, NP}, X32, kch, M);  // g_i C_i d_{i+1}
          }
          each32<C>(M, [&](int j, int q, int r, int cc) {
            const float2 y = ys[i * MAT + r * NP + cc];
            const float2 c1 = i < nlay - 1 ? c.get(j, q) : make_float2(0.f, 0.f);
            const float2 d = make_float2(__fadd_rn(y.x, c1.x), __fadd_rn(y.y, c1.y));
            c.set(j, q, d);
            if (r < n && cc < n) {
              double2& e = X64[(long long)i * MAT + r * NP + cc];
              const double2 x = cadd(e, make_double2((double)d.x, (double)d.y));
              e = x;
              dmax = fmax(dmax, fmax(fabs((double)d.x), fabs((double)d.y)));
              xmax = fmax(xmax, fmax(fabs(x.x), fabs(x.y)));
            }
          });
        }
        if (block_any(!(isfinite(dmax) && isfinite(xmax)))) {
          status = kNonFinite;
          break;
        }
        dmax = block_max(dmax, sh.red);
        xmax = block_max(xmax, sh.red);
        const double nu = xmax > 0.0 ? dmax / xmax : 0.0;
        if (nu <= tol) {
          done = true;
        } else if (it >= 2) {
          const double rho = nu / nu_prev;
          if (rho > 0.5) {
            status = kRefineFail;  // the correction stopped shrinking
            break;
          }
          if (nu * rho <= tol) done = true;
        }
        nu_prev = nu;
      }
      if (status == kOk && !done) status = kRefineFail;
      // 4. Gamma and trace in FP64 from X_0 = G_{0,L-1}.
      __syncthreads();
      if (status == kOk) {
        tval = trace_t<C>(sigL, sigR, X64, GL, U64, n, max(n, max(a.nl, a.nr)), X, sh.red, L);
        if (!isfinite(tval)) status = kNonFinite;
      }
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
      if (steps_out) steps_out[p] = steps;
    }
    __syncthreads();
  }
}

}  // namespace mid
}  // namespace negf
