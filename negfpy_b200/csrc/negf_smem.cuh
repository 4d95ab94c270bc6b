// Building blocks of one (omega, k) point on one thread block -- FP64 products on
// the tensor path and a Gauss-Jordan inverse whose matrix stays in registers -- and
// the kernels of block order n <= 48, with three matrices in shared memory.  The
// kernels up to order 104 (negf_mid.cuh) use the blocks, too.
//
// What bounds these kernels is the FP64 pipe (64 multiply-adds per clock and
// SM, the same for DMMA and DFMA, which share it) and the latency of the n
// dependent pivot steps of each inverse.  One point alone leaves the pipe idle
// through every pivot chain, so several points share an SM: the matrix being
// inverted and all product results live in registers (each thread owns fixed
// elements, see Lane), which leaves three matrices per point in shared memory
// -- 110 KB at n = 48, two points per SM; 31 KB at n = 24, six.
//
// Tiles are 8 x 8 (mma.sync m8n8k4, full rate on sm_100a; m16n8k8 is four of
// them, bit for bit), so orders pad to a multiple of 8 only.
//
// Shared matrices: interleaved (re, im), row-major with row stride NP, the
// column index XOR-swizzled per row (swz): conflict-free for A fragments,
// B fragments, their conjugate transposes, accumulator stores and column walks.
#pragma once
#include "negf_common.cuh"
#include "negf_f64.h"
#include "negf_umma.cuh"

namespace negf {
namespace smem {

// z = (omega + i eta)^2 with the two products rounded separately, as the
// reference's complex power does (no fused multiply-add in the real part).
__device__ __forceinline__ double2 z_of(double w, double e) {
  return make_double2(__dsub_rn(__dmul_rn(w, w), __dmul_rn(e, e)), __dmul_rn(2.0 * w, e));
}

// NP: padded order; each warp owns TR x TC tiles of 8 x 8; OCC: thread blocks
// per SM the registers are budgeted for; KB: bits of the row index in a pivot
// key (6 up to order 48, 8 above); LPR: lanes that share a panel row in the
// pivot steps (0: as many as the threads allow); PARK: column tiles an
// inversion keeps in Tensor Memory during the pivot steps (TR = 1 only), so
// that these do not spill.
template <int NP_, int TR_, int TC_, int OCC_, int KB_ = 6, int LPR_ = 0, int PARK_ = 0>
struct Cfg {
  static constexpr int PARK = PARK_;
  static constexpr int NP = NP_, TR = TR_, TC = TC_, OCC = OCC_, KB = KB_;
  static constexpr int T8 = NP / 8;
  static constexpr int WC = T8 / TC, WR = T8 / TR;
  static constexpr int NW = WR * WC;      // warps
  static constexpr int NTH = 32 * NW;     // threads
  static constexpr int MAT = NP * NP;     // complex elements of a matrix
  // A panel row is handled by LPR neighbouring lanes, EPT columns each: lane cl
  // has columns cl + LPR q.  Rows are PS elements apart, so that the rows of a
  // quarter warp fall into different banks.
  static constexpr int LPR = LPR_ ? LPR_ : (NTH >= 8 * NP ? 8 : (NTH >= 4 * NP ? 4 : 2));
  static constexpr int EPT = 8 / LPR;
  static constexpr int PS = LPR == 8 ? 8 : 8 + LPR;
  static constexpr int PE = NP * PS;      // complex elements of a panel
  // Panel ping-pong and the panel's pivot rows; they share the third matrix
  // buffer (unused while a matrix is inverted) where it is large enough.
  static constexpr int SCR = 2 * PE + 8 * NP;
  static constexpr int BUF = MAT > SCR ? MAT : SCR;
  static_assert(T8 % TR == 0 && T8 % TC == 0 && NP <= (1 << KB) && NW <= 32, "tile split");
  static constexpr int WW = (NP * LPR + 31) / 32;  // warps with panel rows
  static_assert(WW <= NW, "panel rows per warp");
};

// Row-dependent XOR swizzle of the column index (bits 0-2), values
// {0, 5, 2, 7, 1, 4, 3, 6} for r mod 8 = 0..7: with 16-byte elements and phases
// of 8 lanes, rows r, r+1 x 4 columns, 4 rows x 2 columns, rows r, r+1 x even
// columns and 8 rows of one column are all conflict-free.
__device__ __forceinline__ int swz(int r) { return (int)((0xCE1EA8u >> (3 * (r & 7))) & 7u); }
template <int NP>
__device__ __forceinline__ int sidx(int r, int c) { return r * NP + (c ^ swz(r)); }

// Thread's place in the block: element (i, j, q) of its tiles is
// (r0 + 8 i, c0 + 8 j + q), q = 0, 1 -- the accumulator layout of m8n8k4.
struct Lane {
  int g, t, R0, C0;  // lane's group and member; the warp's first row and column
  int r0, c0;        // R0 + g, C0 + 2 t
};
template <class C>
__device__ __forceinline__ Lane lane_geo() {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  Lane L;
  L.g = l >> 2;
  L.t = l & 3;
  L.R0 = (w / C::WC) * C::TR * 8;
  L.C0 = (w % C::WC) * C::TC * 8;
  L.r0 = L.R0 + L.g;
  L.c0 = L.C0 + 2 * L.t;
  return L;
}

// The thread's elements of one matrix.
template <class C>
struct Acc {
  double re[C::TR][C::TC][2], im[C::TR][C::TC][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < C::TR; ++i)
#pragma unroll
      for (int j = 0; j < C::TC; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) re[i][j][q] = im[i][j][q] = 0.0;
  }
  __device__ __forceinline__ double2 get(int i, int j, int q) const { return make_double2(re[i][j][q], im[i][j][q]); }
  __device__ __forceinline__ void set(int i, int j, int q, double2 v) {
    re[i][j][q] = v.x;
    im[i][j][q] = v.y;
  }
};
// f(i, j, q, row, column) over the thread's elements.
template <class C, class F>
__device__ __forceinline__ void each(const Lane& L, F&& f) {
#pragma unroll
  for (int i = 0; i < C::TR; ++i)
#pragma unroll
    for (int j = 0; j < C::TC; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) f(i, j, q, L.r0 + 8 * i, L.c0 + 8 * j + q);
}

// The larger of the high words of |re| and |im|.
__device__ __forceinline__ unsigned hi_word(double2 v) {
  const unsigned ha = (unsigned)__double2hiint(v.x) & 0x7fffffffu;
  const unsigned hb = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
  return ha > hb ? ha : hb;
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Fragments of one chunk of 8 of the contraction (h: its two halves of 4).
// A element (row r0 + 8 i, k); B element (k, column C0 + 8 j + g).  A chunk
// never changes an index modulo 8, so an address is a base per half plus
// constants: row-major walks step by 8, column walks by 8 NP.
template <class C, bool CT>
__device__ __forceinline__ void a_base(const Lane& L, int (&b)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = L.t + 4 * h;
    b[h] = CT ? k * C::NP + L.R0 + (L.g ^ swz(k)) : L.r0 * C::NP + (k ^ swz(L.g));
  }
}
template <class C, bool CT>
__device__ __forceinline__ void b_base(const Lane& L, int (&b)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = L.t + 4 * h;
    b[h] = CT ? (L.C0 + L.g) * C::NP + (k ^ swz(L.g)) : k * C::NP + L.C0 + (L.g ^ swz(k));
  }
}
// Fragments of one row tile of A or one column tile of B.
struct AFrag {
  double re[2], im[2];
};
template <class C, bool CT>
__device__ __forceinline__ void load_a(AFrag& f, const double2* S, const int (&b)[2], int kc, int i) {
  const int off = CT ? kc * 8 * C::NP + 8 * i : kc * 8 + 8 * i * C::NP;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double2 v = S[b[h] + off];
    f.re[h] = v.x;
    f.im[h] = CT ? -v.y : v.y;
  }
}
template <class C, bool CT>
__device__ __forceinline__ void load_b(AFrag& f, const double2* S, const int (&b)[2], int kc, int j) {
  const int off = CT ? kc * 8 + 8 * j * C::NP : kc * 8 * C::NP + 8 * j;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double2 v = S[b[h] + off];
    f.re[h] = v.x;
    f.im[h] = CT ? -v.y : v.y;
  }
}
// One chunk of 8 of one tile: re += ar br, then - ai bi; im += ar bi, then
// ai br (each over its 8 terms in order, as one m16n8k8 per term pair would).
__device__ __forceinline__ void chunk(double (&re)[2], double (&im)[2], const AFrag& a, const AFrag& b) {
  dmma(re, a.re[0], b.re[0]);
  dmma(im, a.re[0], b.im[0]);
  dmma(re, a.re[1], b.re[1]);
  dmma(im, a.re[1], b.im[1]);
  dmma(re, -a.im[0], b.im[0]);
  dmma(im, a.im[0], b.re[0]);
  dmma(re, -a.im[1], b.im[1]);
  dmma(im, a.im[1], b.re[1]);
}

// c1 = op(A1) op(B) and, with two left operands, c2 = op(A2) op(B), over the
// first kch chunks of 8 (the rest is zero padding).  The next row tile's
// fragments, and the next chunk's B, are loaded under the current row's MMAs:
// one or two warps per scheduler do not hide the loads by themselves.
template <class C, int NA, bool AC, bool BC>
__device__ __forceinline__ void mm_(Acc<C>& c1, Acc<C>& c2, const double2* A1, const double2* A2, const double2* B,
                                    int kch, const Lane& L) {
  int ab[2], bb[2];
  a_base<C, AC>(L, ab);
  b_base<C, BC>(L, bb);
  c1.zero();
  if (NA == 2) c2.zero();
  AFrag a, an, b[C::TC], bn[C::TC];
#pragma unroll
  for (int j = 0; j < C::TC; ++j) load_b<C, BC>(b[j], B, bb, 0, j);
  load_a<C, AC>(a, A1, ab, 0, 0);
#pragma unroll 1
  for (int kc = 0; kc < kch; ++kc) {
    const int kn = kc + 1 < kch ? kc + 1 : 0;
#pragma unroll
    for (int r = 0; r < NA * C::TR; ++r) {
      const int i = r % C::TR, rn = r + 1;
      if (rn < NA * C::TR) load_a<C, AC>(an, rn < C::TR ? A1 : A2, ab, kc, rn % C::TR);
      else load_a<C, AC>(an, A1, ab, kn, 0);
      if (r == 0) {
#pragma unroll
        for (int j = 0; j < C::TC; ++j) load_b<C, BC>(bn[j], B, bb, kn, j);
      }
      Acc<C>& c = r < C::TR ? c1 : c2;
#pragma unroll
      for (int j = 0; j < C::TC; ++j) chunk(c.re[i][j], c.im[i][j], a, b[j]);
      a = an;
    }
#pragma unroll
    for (int j = 0; j < C::TC; ++j) b[j] = bn[j];
  }
}
template <class C, bool AC, bool BC>
__device__ __forceinline__ void mm(Acc<C>& c, const double2* A, const double2* B, int kch, const Lane& L) {
  mm_<C, 1, AC, BC>(c, c, A, A, B, kch, L);
}
template <class C>
__device__ __forceinline__ void mm2(Acc<C>& c1, Acc<C>& c2, const double2* A1, const double2* A2, const double2* B,
                                    int kch, const Lane& L) {
  mm_<C, 2, false, false>(c1, c2, A1, A2, B, kch, L);
}
template <class C>
__device__ __forceinline__ void store_acc(double2* S, const Acc<C>& c, const Lane& L) {
  each<C>(L, [&](int i, int j, int q, int r, int cc) { S[sidx<C::NP>(r, cc)] = c.get(i, j, q); });
}
// Global nr x nc row-major matrix -> padded shared buffer (zeros outside).
template <class C>
__device__ __forceinline__ void load_mat(double2* S, const double2* __restrict__ G, int nr, int nc) {
  for (int idx = threadIdx.x; idx < C::MAT; idx += C::NTH) {
    const int r = idx / C::NP, c = idx - r * C::NP;
    S[sidx<C::NP>(r, c)] = (r < nr && c < nc) ? G[(long long)r * nc + c] : make_double2(0.0, 0.0);
  }
}

// 1 / (a + ib) by Smith's algorithm (R. L. Smith, CACM 5(8), 1962).
__device__ __forceinline__ double2 crecip_smith(double2 v) {
  if (fabs(v.x) >= fabs(v.y)) {
    const double r = v.y / v.x;
    const double i = 1.0 / fma(v.y, r, v.x);
    return make_double2(i, -r * i);
  }
  const double r = v.x / v.y;
  const double i = 1.0 / fma(v.x, r, v.y);
  return make_double2(r * i, -i);
}

// ---------------------------------------------------- thread-private matrices --
// A matrix that only its owning threads touch (eps, eps_s) lives in Tensor
// Memory: tile (i, j) of a thread is 8 consecutive columns of its lane, so that
// it costs neither registers nor shared memory, and, unlike local memory
// (measured: the few KB of L1 beside 222 KB of shared memory send it to L2),
// it is a few cycles away.  Warp w holds lanes 32 (w % 4); the warps beyond
// four use further columns.
template <class C>
struct Tmem {
  static constexpr int kMat = C::TR * C::TC * 8;                  // columns of one matrix
  static constexpr int kNeed = (C::NW + 3) / 4 * 2 * kMat;        // two matrices, every warp
  static constexpr int kCols = kNeed <= 32 ? 32 : kNeed <= 64 ? 64 : kNeed <= 128 ? 128 : 256;
  static_assert(kNeed <= 256, "TMEM columns");
};
__device__ __forceinline__ void tmem_put(uint32_t addr, const double2 (&v)[2]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr),
               "r"(__double2loint(v[0].x)), "r"(__double2hiint(v[0].x)), "r"(__double2loint(v[0].y)),
               "r"(__double2hiint(v[0].y)), "r"(__double2loint(v[1].x)), "r"(__double2hiint(v[1].x)),
               "r"(__double2loint(v[1].y)), "r"(__double2hiint(v[1].y))
               : "memory");
}
__device__ __forceinline__ void tmem_stored() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// N tiles from consecutive addresses (the loads are in flight together).
template <int N>
__device__ __forceinline__ void tmem_get(uint32_t addr, double2 (&v)[N][2]) {
  int r[N][8];
#pragma unroll
  for (int i = 0; i < N; ++i)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[i][0]), "=r"(r[i][1]), "=r"(r[i][2]), "=r"(r[i][3]), "=r"(r[i][4]), "=r"(r[i][5]),
                   "=r"(r[i][6]), "=r"(r[i][7])
                 : "r"(addr + 8 * i));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) {  // keeps every use behind the wait
    asm volatile(""
                 : "+r"(r[i][0]), "+r"(r[i][1]), "+r"(r[i][2]), "+r"(r[i][3]), "+r"(r[i][4]), "+r"(r[i][5]),
                   "+r"(r[i][6]), "+r"(r[i][7]));
#pragma unroll
    for (int q = 0; q < 2; ++q)
      v[i][q] = make_double2(__hiloint2double(r[i][4 * q + 1], r[i][4 * q]),
                             __hiloint2double(r[i][4 * q + 3], r[i][4 * q + 2]));
  }
}

// f(j, elements) for tiles 0 .. N-1 at consecutive addresses, four in flight.
template <int N, class F>
__device__ __forceinline__ void tmem_tiles(uint32_t addr, F&& f) {
#pragma unroll
  for (int j = 0; j + 4 <= N; j += 4) {
    double2 v[4][2];
    tmem_get<4>(addr + 8 * j, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) f(j + i, v[i]);
  }
  if (N % 4) {
    constexpr int R = N % 4 ? N % 4 : 1;
    double2 v[R][2];
    tmem_get<R>(addr + 8 * (N - R), v);
#pragma unroll
    for (int i = 0; i < R; ++i) f(N - R + i, v[i]);
  }
}

// ---------------------------------------------------------- Gauss-Jordan --
template <class C>
struct GJ {
  alignas(16) double2 lam[2];          // the panel's scale, double-buffered by column parity
  alignas(16) unsigned key[8][C::NW];  // each warp's pivot key of each panel column
  int fail;                            // status of the panel's pivots
  int newpos[C::NP];                   // position after the panel of each panel row
  int cmapinv[C::NP];
};

// Pivot key of a candidate entry: top bits of max(|re|, |im|) with the row
// index in the low KB bits, so the unsigned maximum over a column picks the
// largest entry up to a relative 2^-14 (KB = 6; 2^-12 for 8), ties to the
// lowest row.
template <int KB>
__device__ __forceinline__ unsigned pivot_key(double2 v, int r) {
  constexpr unsigned M = (1u << KB) - 1u;
  return (hi_word(v) & ~M) | (M - (unsigned)r);
}

// Inverse of the matrix held in m (leading n x n block, identity padding) by
// blocked Gauss-Jordan elimination with partial pivoting, into the shared
// matrix out; scr (SCR complex, may be out itself) is scratch, park the thread's
// TMEM columns for C::PARK tiles.  Ends with the
// block synchronised.
//
// Columns are processed in panels of 8.  The n x 8 panel is factored in shared
// memory by the whole block with one barrier per column and no division: it is
// kept as W = lambda P (P the textbook Gauss-Jordan panel, lambda a complex
// scalar) and, with p the pivot and s a power of two bringing p near 1,
//     new(r, c) = (p s) a' - (s b') m,   lambda <- lambda p s
//     a' = 0 if r is the pivot row or c the pivot column, else W(r, c)
//     b' = -lambda for the pivot row, else W(r, j)
//     m  =  lambda for the pivot column, else W(pivot row, c)
// (expanding W = lambda P gives the textbook update times the new lambda;
// |p s| lies in [1, 2.83]).  Pivot search is looked ahead: the threads that
// write column j+1 of the panel reduce its pivot keys (see pivot_key) over the
// rows not yet used as pivots, one slot per warp, before the barrier; the key's
// exponent bits give s.
//
// The matrix itself never moves: a thread keeps its elements in registers for
// the whole inversion and only tracks the position of its rows.  It writes its
// part of the panel's 8 columns to shared memory at those positions, and its
// part of the pivot rows once they are known; the rank-8 update then
// accumulates in place on the tensor path,
//     row r, columns Q: [r not a pivot row] W(r, Q) + P(r, :) W(pivot rows, Q),
//     row r, panel:     P(r, :),                      P = W / lambda.
// The row order and the undone column interchanges (column c of the inverse is
// column t_{n-1}(...t_0(c)) of the eliminated matrix, t_k = (k b_k), b_k the
// position of the k-th pivot) are applied as the result is written.  Keeping
// the matrix in registers instead of two shared buffers removes its reload and
// rewrite in each of the n/8 updates and is what lets several points share an SM.
// Returns kOk, kSingular (all candidates zero or below 2^-1022) or kNonFinite
// identically in every thread.
template <class C>
__device__ __forceinline__ int gj_invert(Acc<C>& m, double2* scr, double2* out, int n, const Lane& L, GJ<C>& sh,
                                         uint32_t park = 0) {
  constexpr int PE = C::PE, NP = C::NP, NW = C::NW;
  constexpr int LPR = C::LPR, EPT = C::EPT, PS = C::PS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool work = C::NW == C::WW || warp < C::WW;              // the warp has panel rows
  const bool live = C::NTH == NP * LPR || tid < NP * LPR;        // the thread has one
  const int pr_own = live ? tid / LPR : 0, cl = tid % LPR;
  const int prow = pr_own * PS;
  double2* const Bp = scr + 2 * PE;  // the panel's pivot rows [8][NP]
  int pos[C::TR];  // position of each of the thread's matrix rows
#pragma unroll
  for (int i = 0; i < C::TR; ++i) pos[i] = L.r0 + 8 * i;
  // The last warp (without panel rows where the block has warps to spare)
  // keeps lambda and the permutations: lane l those of rows and columns l,
  // l + 32, ...
  const bool bk = warp == NW - 1;
  constexpr bool kSpare = NW > C::WW;
  constexpr bool kAll = NW <= C::WW + 1;  // every warp takes part in the pivot steps
  constexpr unsigned kRow = (1u << C::KB) - 1u;
  constexpr int RL = (NP + 31) / 32;
  int cm[RL];  // t_k(...t_0(c)) over the steps done so far
#pragma unroll
  for (int i = 0; i < RL; ++i) cm[i] = lane + 32 * i;

#pragma unroll 1
  for (int k0 = 0, par = 0; k0 < n; k0 += 8, par ^= 1) {
    const int jmax = (n - k0) < 8 ? (n - k0) : 8;
    // A full panel's 8 steps end in the buffer they began in, so the next
    // panel starts in the other one while this one may still be read.
    double2* const P0 = scr + par * PE;
    double2* const P1 = scr + (par ^ 1) * PE;
    const int pj = (k0 - L.C0) >> 3;  // the panel's tile column among the thread's, if in range
    // ---- publish the panel, keys of panel column 0 ----
    unsigned key0 = 0u;
#pragma unroll
    for (int j = 0; j < C::TC; ++j)
      if (j == pj) {
#pragma unroll
        for (int i = 0; i < C::TR; ++i) {
          double2* row = P0 + pos[i] * PS + 2 * L.t;
          row[0] = m.get(i, j, 0);
          row[1] = m.get(i, j, 1);
          if (L.t == 0 && pos[i] >= k0 && pos[i] < n) key0 = max(key0, pivot_key<C::KB>(m.get(i, j, 0), pos[i]));
        }
      }
    key0 = __reduce_max_sync(0xffffffffu, key0);
    if (lane == 0) sh.key[0][warp] = key0;
    if (tid == 0) sh.lam[0] = make_double2(1.0, 0.0);
    __syncthreads();
    if (C::PARK) {
#pragma unroll
      for (int j = 0; j < C::PARK; ++j) {
        const int jj = C::TC - C::PARK + j;
        const double2 v[2] = {m.get(0, jj, 0), m.get(0, jj, 1)};
        tmem_put(park + 8 * j, v);
      }
      tmem_stored();
    }
    // ---- factor the panel, one barrier per column, by the warps with panel
    // rows and the bookkeeping warp; the others wait for the panel ----
    if (work || bk) {
      double2 av[EPT];  // this thread's panel elements
#pragma unroll
      for (int q = 0; q < EPT; ++q) av[q] = P0[prow + cl + LPR * q];
      bool cand = live && pr_own >= k0 && pr_own < n;  // row not yet a pivot
      int fail = kOk;  // the first bad pivot's status
      int lg[RL];                                      // position of panel rows lane + 32 i
#pragma unroll
      for (int i = 0; i < RL; ++i) lg[i] = lane + 32 * i;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= jmax) break;
        const double2* Pc = (j & 1) ? P1 : P0;
        double2* Pn = (j & 1) ? P0 : P1;
        // What does not depend on the pivot is loaded with the key (one slot per
        // warp; after the panel's first column only warps with rows post one).
        const double2 fv = Pc[prow + j];
        const double2 lam = sh.lam[j & 1];
        unsigned key;
        if (NW == 4 && kAll) {  // every slot is posted in every step
          const uint4 kv = *reinterpret_cast<const uint4*>(sh.key[j]);
          key = max(max(kv.x, kv.y), max(kv.z, kv.w));
        } else if (NW == 2 && kAll) {
          const uint2 kv = *reinterpret_cast<const uint2*>(sh.key[j]);
          key = max(kv.x, kv.y);
        } else if (NW == 1) {
          key = sh.key[j][0];
        } else {
          key = __reduce_max_sync(0xffffffffu, lane < (j == 0 ? NW : C::WW) ? sh.key[j][lane] : 0u);
        }
        // A zero or non-finite pivot ends the inversion at the end of the panel
        // (off the path to the pivot row); min keeps its row in the panel.
        const bool stop = key - (kRow + 1u) >= 0x7ff00000u - (kRow + 1u);
        const int pr = min((int)(kRow - (key & kRow)), NP - 1);
        const int ex = (int)(key >> 20);
        const double sc = (ex != 0 && ex < 2046) ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
        const double2* prow_p = Pc + pr * PS;
        const double2 piv = prow_p[j];
        const double2 ps = make_double2(piv.x * sc, piv.y * sc);
        unsigned nk = 0u;
        if (work) {
          double2 mv[EPT];
#pragma unroll
          for (int q = 0; q < EPT; ++q) mv[q] = prow_p[cl + LPR * q];
          const bool isp = pr_own == pr;
          cand = cand && !isp;
          const double2 bb = isp ? lam : fv;
          const double nsc = isp ? sc : -sc;
          const double2 nb = make_double2(bb.x * nsc, bb.y * nsc);  // -s b', so that nothing is negated below
          const double2 pe = isp ? make_double2(0.0, 0.0) : ps;  // no branch: a' = 0 as a zero factor
          // The next pivot column first, so that its keys are reduced under the
          // other columns' updates.
#pragma unroll
          for (int qq = 0; qq < EPT; ++qq) {
            const int q = (qq + (j + 1) / LPR) % EPT;
            const int c = cl + LPR * q;
            const bool pivcol = q == j / LPR && cl == j % LPR;
            const double2 mq = pivcol ? lam : mv[q];
            double2 v = make_double2(fma(nb.x, mq.x, -nb.y * mq.y), fma(nb.x, mq.y, nb.y * mq.x));
            cfma(v, pivcol ? make_double2(0.0, 0.0) : pe, av[q]);
            if (live) Pn[prow + c] = v;
            av[q] = v;
            if (j + 1 < 8 && qq == 0) {
              if (cl == (j + 1) % LPR && cand) nk = pivot_key<C::KB>(v, pr_own);
              nk = __reduce_max_sync(0xffffffffu, nk);
            }
          }
        }
        if (j + 1 < 8 && lane == 0) sh.key[j + 1][warp] = nk;
        if (bk) {
          double2 ln = cmul(lam, ps);
          if (kSpare && j == 7) ln = crecip_smith(ln);  // under the other warps' element updates
          if (lane == 0) sh.lam[(j + 1) & 1] = ln;
          // the row interchange of this step: positions k and bl
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
        if (stop) fail = fail ? fail : (key <= kRow ? kSingular : kNonFinite);
        if (j + 1 < jmax) {
          if (kAll) __syncthreads();
          else asm volatile("bar.sync 1, %0;" ::"n"(32 * (C::WW + 1)) : "memory");
        }
      }
      if (bk && lane == 0) sh.fail = fail;
    }
    __syncthreads();
    // ---- rank-8 update in registers ----
    if (sh.fail) return sh.fail;
    if (C::PARK) {
      double2 v[C::PARK ? C::PARK : 1][2];
      tmem_get<C::PARK ? C::PARK : 1>(park, v);
#pragma unroll
      for (int j = 0; j < C::PARK; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) m.set(0, C::TC - C::PARK + j, q, v[j][q]);
    }
    // The owners of the pivot rows hand out their elements before the panel.
    int np[C::TR];
#pragma unroll
    for (int i = 0; i < C::TR; ++i) np[i] = sh.newpos[pos[i]];
#pragma unroll
    for (int i = 0; i < C::TR; ++i) {
      if ((unsigned)(np[i] - k0) < (unsigned)jmax) {
        double2* row = Bp + (np[i] - k0) * NP;
        const int sw = swz(np[i]);
#pragma unroll
        for (int j = 0; j < C::TC; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            row[L.C0 + 8 * j + ((2 * L.t + q) ^ sw)] = m.get(i, j, q);
            m.set(i, j, q, make_double2(0.0, 0.0));
          }
      }
    }
    const double2* P = (jmax & 1) ? P1 : P0;
    const double2 ll = sh.lam[jmax & 1];
    const double2 il = kSpare && jmax == 8 ? ll : crecip_smith(ll);
    AFrag a[C::TR];
#pragma unroll
    for (int i = 0; i < C::TR; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 v = cmul(P[pos[i] * PS + L.t + 4 * h], il);
        a[i].re[h] = v.x;
        a[i].im[h] = v.y;
      }
    __syncthreads();
    auto pivots = [&](AFrag& b, int j) {  // column tile j of the pivot rows
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int kk = L.t + 4 * h;
        const double2 v = Bp[sidx<NP>(kk, L.C0 + 8 * j + L.g)];
        b.re[h] = kk < jmax ? v.x : 0.0;
        b.im[h] = kk < jmax ? v.y : 0.0;
      }
    };
    AFrag b, bn;
    pivots(b, 0);
#pragma unroll
    for (int j = 0; j < C::TC; ++j) {
      if (j + 1 < C::TC) pivots(bn, j + 1);
      if (j == pj) {  // the panel's columns take P(r, :) (warp-uniform)
#pragma unroll
        for (int i = 0; i < C::TR; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q) m.set(i, j, q, cmul(P[pos[i] * PS + 2 * L.t + q], il));
      } else {
#pragma unroll
        for (int i = 0; i < C::TR; ++i) chunk(m.re[i][j], m.im[i][j], a[i], b);
      }
      b = bn;
    }
#pragma unroll
    for (int i = 0; i < C::TR; ++i) pos[i] = np[i];
  }
  if (bk)
#pragma unroll
    for (int i = 0; i < RL; ++i)
      if (lane + 32 * i < NP) sh.cmapinv[cm[i]] = lane + 32 * i;
  __syncthreads();  // the last panel and its pivot rows are read, cmapinv is complete
#pragma unroll
  for (int j = 0; j < C::TC; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = sh.cmapinv[L.c0 + 8 * j + q];
#pragma unroll
      for (int i = 0; i < C::TR; ++i) out[sidx<NP>(pos[i], c)] = m.get(i, j, q);
    }
  __syncthreads();
  return kOk;
}

// Shared memory of a point: alpha, beta (or g, G0) and the third buffer, the
// inversion's bookkeeping, reduction slots.
template <class C>
struct Shared {
  GJ<C> gj;
  double red[40];
  uint32_t tmem;
};
template <class C>
constexpr size_t shared_bytes() { return (size_t)(2 * C::MAT + C::BUF) * 16 + sizeof(Shared<C>); }

// ------------------------------------------------------------ Sancho-Rubio --
// alpha in A, beta in B, g and then alpha g and beta g in X; eps and eps_s, which
// only the thread that owns an element touches, in Tensor Memory.
template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) sr_f64_kernel(SrArgs a) {
  constexpr int MAT = C::MAT, NP = C::NP;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const A = reinterpret_cast<double2*>(smraw);
  double2* const B = A + MAT;
  double2* const X = B + MAT;
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);

  const int p = blockIdx.x;
  if (p >= a.batch) return;
  const int n = a.n;
  const int kch = (n + 7) >> 3;
  const int tid = threadIdx.x;
  const Lane L = lane_geo<C>();
  const long long kset = a.kidx ? (long long)a.kidx[p] : 0;
  const double2* h00 = a.h00 + kset * a.lead_stride;
  const double2* h01 = a.h01 + kset * a.lead_stride;
  const double2* h10 = a.h10 ? a.h10 + kset * a.lead_stride : nullptr;
  const double w = a.omega[p];
  const double2 z = z_of(w, a.eta[p]);

  if (tid < 32) umma::tmem_alloc(&sh.tmem, Tmem<C>::kCols);
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t eps = sh.tmem + ((uint32_t)(tid >> 5 & 3) << 21) + (uint32_t)(tid >> 7) * 2 * Tmem<C>::kMat;
  const uint32_t es = eps + Tmem<C>::kMat;
#pragma unroll
  for (int i = 0; i < C::TR; ++i)
#pragma unroll
    for (int j = 0; j < C::TC; ++j) {
      double2 v[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = L.r0 + 8 * i, c = L.c0 + 8 * j + q;
        v[q] = (r < n && c < n) ? h00[r * n + c] : make_double2(0.0, 0.0);
      }
      tmem_put(eps + (i * C::TC + j) * 8, v);
      tmem_put(es + (i * C::TC + j) * 8, v);
    }
  for (int idx = tid; idx < MAT; idx += C::NTH) {
    const int r = idx / NP, c = idx - r * NP;
    const bool in = r < n && c < n;
    A[sidx<NP>(r, c)] = in ? h01[r * n + c] : make_double2(0.0, 0.0);
    B[sidx<NP>(r, c)] = in ? (h10 ? h10[r * n + c] : cconj(h01[c * n + r])) : make_double2(0.0, 0.0);
  }
  // m = z - e on the leading block, identity in the padding
  auto form = [&](Acc<C>& m, uint32_t e) {
    tmem_stored();
#pragma unroll
    for (int i = 0; i < C::TR; ++i) {
      double2 x[C::TC][2];
      tmem_get<C::TC>(e + i * C::TC * 8, x);
#pragma unroll
      for (int j = 0; j < C::TC; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int r = L.r0 + 8 * i, c = L.c0 + 8 * j + q;
          double2 v;
          if (r < n && c < n) v = (r == c) ? csub(z, x[j][q]) : cneg(x[j][q]);
          else v = make_double2(r == c ? 1.0 : 0.0, 0.0);
          m.set(i, j, q, v);
        }
    }
  };
  // e += d; returns the largest high word (non-finite from 0x7ff00000 on)
  auto add = [&](uint32_t e, const Acc<C>& d) {
    unsigned hi = 0u;
    tmem_stored();
#pragma unroll
    for (int i = 0; i < C::TR; ++i) {
      double2 x[C::TC][2];
      tmem_get<C::TC>(e + i * C::TC * 8, x);
#pragma unroll
      for (int j = 0; j < C::TC; ++j) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          x[j][q] = cadd(x[j][q], d.get(i, j, q));
          hi = max(hi, hi_word(x[j][q]));
        }
        tmem_put(e + (i * C::TC + j) * 8, x[j]);
      }
    }
    return hi;
  };
  // The largest high word of a new alpha or beta, and whether an element's
  // magnitude is tol or more.  A component above tol decides that by its high
  // word alone (its square is then at least tol^2 in any rounding).
  const double tol2 = a.tol * a.tol;
  const unsigned htol = (unsigned)__double2hiint(a.tol);
  auto measure = [&](const Acc<C>& d, unsigned& hi, int& big) {
    unsigned h = 0u;
    each<C>(L, [&](int i, int j, int q, int, int) { h = max(h, hi_word(d.get(i, j, q))); });
    hi = max(hi, h);
    if (h > htol) {
      big = 1;
    } else {
      each<C>(L, [&](int i, int j, int q, int, int) { big |= !(cabs2(d.get(i, j, q)) < tol2); });
    }
  };

  int status = kOk;
  int it = 0;  // sweeps begun
  Acc<C> c1, c2;
  bool converged = false;
  for (;;) {
    // (z - eps)^-1, or the surface GF (z - eps_s)^-1 once converged
    if (!converged) ++it;
    form(c1, converged ? es : eps);
    status = gj_invert<C>(c1, X, X, n, L, sh.gj);
    if (status != kOk || converged) break;
    // alpha g, beta g
    mm2<C>(c1, c2, A, B, X, kch, L);
    __syncthreads();
    store_acc<C>(X, c1, L);
    __syncthreads();
    // eps_s += (alpha g) beta, eps += (alpha g) beta
    unsigned hi = 0u;
    int big = 0;
    mm<C, false, false>(c1, X, B, kch, L);
    hi = add(es, c1);
    add(eps, c1);
    // alpha' = (alpha g) alpha, kept in registers while alpha is still needed
    mm<C, false, false>(c1, X, A, kch, L);
    measure(c1, hi, big);
    __syncthreads();
    store_acc<C>(X, c2, L);
    __syncthreads();
    // eps += (beta g) alpha
    mm<C, false, false>(c2, X, A, kch, L);
    hi = max(hi, add(eps, c2));
    // beta' = (beta g) beta
    mm<C, false, false>(c2, X, B, kch, L);
    measure(c2, hi, big);
    const int any_bad = block_any(hi >= 0x7ff00000u);  // a barrier: every read of alpha, beta and X is done
    store_acc<C>(A, c1, L);
    store_acc<C>(B, c2, L);
    if (any_bad) {
      status = sr_failure_status(it, n, h00, h01, h10, z);
      break;
    }
    converged = !block_any(big);  // max(|alpha|, |beta|) < tol
    if (!converged && it == a.maxiter) {
      status = kMaxIter;
      break;
    }
  }
  tmem_stored();
  __syncthreads();
  if (tid < 32) umma::tmem_dealloc(sh.tmem, Tmem<C>::kCols);
  if (status == kOk) {
    if (a.g_out) {
      double2* go = a.g_out + (long long)p * n * n;
      for (int idx = tid; idx < n * n; idx += C::NTH) {
        const int r = idx / n, c = idx - r * n;
        go[idx] = X[sidx<NP>(r, c)];
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
}

// ---------------------------------------------------------------- RGF sweep --
// X: g of the layer before, then W = g C, then the inversion's scratch and the
// new g; Y: G_{0,l-1}, then U = G_{0,l-1} C, then G_{0,l}; Cb: the coupling C.
// Sigma_L and Sigma_R of the point in the block's global scratch.
template <class C>
__global__ void __launch_bounds__(C::NTH, C::OCC) rgf_f64_kernel(RgfArgs a) {
  constexpr int MAT = C::MAT, NP = C::NP;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* const Cb = reinterpret_cast<double2*>(smraw);
  double2* const Y = Cb + MAT;
  double2* const X = Y + MAT;
  Shared<C>& sh = *reinterpret_cast<Shared<C>*>(X + C::BUF);
  __shared__ int s_point;

  const int n = a.n, nlay = a.L;
  const int kch = (n + 7) >> 3;
  const int tid = threadIdx.x;
  const Lane L = lane_geo<C>();
  double2* sigL = a.sigma_ws + (long long)blockIdx.x * 2 * n * n;
  double2* sigR = sigL + (long long)n * n;
  Acc<C> c1, c2;

  for (;;) {
    if (tid == 0) s_point = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int p = s_point;
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

    // Contact self-energies Sigma = V g V^H into this block's scratch.
    for (int side = 0; side < 2; ++side) {
      const int nl = side ? a.nr : a.nl;
      const int lch = (nl + 7) >> 3;
      const double2* V = side ? a.VR + k * a.vr_ks : a.VL + k * a.vl_ks;
      const double2* g = side ? a.gR + (long long)p * a.gr_ps : a.gL + (long long)p * a.gl_ps;
      double2* S = side ? sigR : sigL;
      load_mat<C>(Cb, V, n, nl);
      load_mat<C>(X, g, nl, nl);
      __syncthreads();
      mm<C, false, false>(c1, Cb, X, lch, L);
      store_acc<C>(Y, c1, L);
      __syncthreads();
      mm<C, false, true>(c1, Y, Cb, lch, L);
      each<C>(L, [&](int i, int j, int q, int r, int c) {
        if (r < n && c < n) S[r * n + c] = c1.get(i, j, q);
      });
      __syncthreads();
    }

    int status = kOk;
    for (int l = 0; l < nlay; ++l) {
      if (l > 0) {
        // identical layers (layer stride 0) share one C: load it once per point
        if (l == 1 || a.c_ls != 0) load_mat<C>(Cb, Cg + (long long)(l - 1) * a.c_ls, n, n);
        __syncthreads();
        // W = g_{l-1} C, U = G_{0,l-1} C
        mm2<C>(c1, c2, X, Y, Cb, kch, L);
        __syncthreads();
        store_acc<C>(X, c1, L);
        store_acc<C>(Y, c2, L);
        __syncthreads();
        mm<C, true, false>(c1, Cb, X, kch, L);  // C^H W
      }
      // M = z - D_l - (C^H W, or Sigma_L on layer 0) [- Sigma_R on the last layer], identity padding
      const double2* Dl = D + (long long)l * a.d_ls;
      each<C>(L, [&](int i, int j, int q, int r, int c) {
        double2 v;
        if (r < n && c < n) {
          v = csub(cneg(Dl[r * n + c]), l == 0 ? sigL[r * n + c] : c1.get(i, j, q));
          if (l == nlay - 1) v = csub(v, sigR[r * n + c]);
          if (r == c) v = cadd(v, z);
        } else {
          v = make_double2(r == c ? 1.0 : 0.0, 0.0);
        }
        c1.set(i, j, q, v);
      });
      __syncthreads();  // every read of W is done
      status = gj_invert<C>(c1, X, X, n, L, sh.gj);
      if (status != kOk) break;
      // G_{0,0} = g_0, G_{0,l} = U g_l
      if (l == 0) {
        each<C>(L, [&](int, int, int, int r, int c) { Y[sidx<NP>(r, c)] = X[sidx<NP>(r, c)]; });
      } else {
        mm<C, false, false>(c1, Y, X, kch, L);
        __syncthreads();
        store_acc<C>(Y, c1, L);
      }
    }
    __syncthreads();
    double tval = 0.0;
    if (status == kOk) {
      // T = Re sum_ij (Gamma_L G Gamma_R)_ij conj(G)_ij, Gamma = i (Sigma - Sigma^H), G = G_{0,L-1} in Y.
      each<C>(L, [&](int, int, int, int r, int c) {
        double2 gl = make_double2(0.0, 0.0), gr = gl;
        if (r < n && c < n) {
          double2 d = csub(sigL[r * n + c], cconj(sigL[c * n + r]));
          gl = make_double2(-d.y, d.x);
          d = csub(sigR[r * n + c], cconj(sigR[c * n + r]));
          gr = make_double2(-d.y, d.x);
        }
        X[sidx<NP>(r, c)] = gl;
        Cb[sidx<NP>(r, c)] = gr;
      });
      __syncthreads();
      mm<C, false, false>(c1, X, Y, kch, L);
      __syncthreads();
      store_acc<C>(X, c1, L);
      __syncthreads();
      mm<C, false, false>(c1, X, Cb, kch, L);
      __syncthreads();
      // The terms are summed in an order that does not depend on the tile
      // split: by 16 x 16 squares, lane (g, t) of a warp adding the elements
      // (g + 8 a, 8 j + 2 t + b) of one square.
      double* terms = reinterpret_cast<double*>(X);
      each<C>(L, [&](int i, int j, int q, int r, int c) {
        const double2 g = Y[sidx<NP>(r, c)];
        double t = 0.0;
        t += c1.re[i][j][q] * g.x + c1.im[i][j][q] * g.y;
        terms[r * NP + c] = t;
      });
      __syncthreads();
      constexpr int T16 = (NP + 15) / 16;
      for (int s = tid >> 5; s < T16 * T16; s += C::NW) {
        double t = 0.0;
        for (int e = 0; e < 8; ++e) {
          const int r = (s / T16) * 16 + L.g + 8 * ((e >> 1) & 1), c = (s % T16) * 16 + 8 * (e >> 2) + 2 * L.t + (e & 1);
          if (r < NP && c < NP) t += terms[r * NP + c];
        }
        t = warp_sum(t);
        if ((tid & 31) == 0) sh.red[s] = t;
      }
      __syncthreads();
      if (tid < 32) {
        tval = warp_sum(tid < T16 * T16 ? sh.red[tid] : 0.0);
        if (!isfinite(tval)) status = kNonFinite;
      }
    }
    if (tid == 0) {
      a.T_out[p] = (status == kOk) ? tval : __longlong_as_double(0x7ff8000000000000ULL);
      if (a.status_out) a.status_out[p] = status;
    }
    __syncthreads();
  }
}

}  // namespace smem
}  // namespace negf
