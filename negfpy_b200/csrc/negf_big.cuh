// FP64 building blocks for one (omega, k) point of order 105..256 on one thread
// block (and, in the uneven batch, of any order): every matrix lives in the
// block's global workspace, column strips of 32 of the matrix at work in
// registers.
//
// A matrix of these orders (0.2-1 MB) fits neither the registers nor the shared
// memory of an SM.  The kernels before this design read both operands of every
// 16 x 16 tile through L1/L2 (32 bytes per clock and SM at full FP64 rate) and
// streamed the whole matrix through L2 in each of the n / 8 updates of an
// inverse (64 bytes per clock and SM): about half the FP64 pipe.  Here warp w
// owns rows 16 w .. 16 w + 15.  A product keeps a 32-column strip of its result
// in registers and takes both operands through a ring in shared memory, filled by
// cp.async four chunks ahead (at full FP64 rate 8 bytes per clock and SM of the left
// one, 256 / n of the right one).  An inverse factors 32 columns at a
// time in registers and applies their four updates to each other strip in one
// pass over it, so that the matrix crosses L2 n / 32 times.
// Decimation / 6-layer sweep at n = 192, ms, before and after: 148 points 109 / 24.8
// -> 51.8 / 10.8, 296 points 125 / 27.5 -> 98.6 / 21.6 (products at 0.77 of the FP64
// pipe, the inverse's strips at 0.45, its pivot steps latency).
// Every element keeps its sequence of operations (chunks of 8, panels of 8), so
// results are bitwise those of the kernels of the smaller orders.
#pragma once
#include "negf_common.cuh"
#include "negf_f64.h"
#include "negf_mid.cuh"
#include "negf_smem.cuh"

namespace negf {
namespace big {

using mid::gamma_of;
using mid::Left;
using smem::AFrag;
using smem::chunk;
using smem::crecip_smith;
using smem::swz;
using smem::z_of;

struct Tiles {
  static constexpr int TR = 2, TC = 4;  // a warp's 8 x 8 tiles of a strip
};
using Acc = smem::Acc<Tiles>;
constexpr int kTC = Tiles::TC, kStrip = 8 * kTC;
// Chunks of both operands in a stage of the products' ring, and stages: two blocks
// per SM have room for five chunks each, one block for six, which halves its
// barriers.
template <int CH>
constexpr int kRing = CH == 1 ? 5 : 3;
constexpr int kMaxWarps = 16;
constexpr int PS = 10;                 // panel row stride: rows of a quarter warp in different banks

// Thread's place: warps 0 .. NP / 16 - 1 own rows; the others only help with
// the copies.  Element (i, j, q) of strip st is (r0 + 8 i, 32 st + 8 j + 2 t + q).
struct Geo {
  int NP, tid, nthr, warp, lane, g, t, r0;
  bool active;
  __device__ __forceinline__ explicit Geo(int np) {
    NP = np;
    tid = threadIdx.x;
    nthr = blockDim.x;
    warp = tid >> 5;
    lane = tid & 31;
    g = lane >> 2;
    t = lane & 3;
    r0 = 16 * warp + g;
    active = 16 * warp < np;
  }
};
struct Ctl {
  alignas(16) double2 lam[2];
  unsigned key[8][kMaxWarps];
  double red[40];
  alignas(16) int pivot[8];   // the panel's pivot rows, by their position before its steps
  int prow[kStrip];           // rows of the pivots of the four panels
  int cinv[256];              // column of the inverse that a column of the eliminated matrix becomes
  int fail, point;
};
// Shared memory: the products' ring, or the inverse's panel pair (later two
// strips' pivot rows), left factors of four panels and a panel's pivot rows;
// then Ctl.
__host__ __device__ constexpr int pair_elems(int np) {
  return 2 * np * PS > 2 * kStrip * kStrip ? 2 * np * PS : 2 * kStrip * kStrip;
}
template <int CH>
__host__ __device__ constexpr size_t region_bytes(int np) {
  const size_t ring = (size_t)kRing<CH> * CH * (8 * np + 8 * kStrip) * 16;
  const size_t gj = ((size_t)pair_elems(np) + 32 * np + 8 * kStrip) * 16;
  return ring > gj ? ring : gj;
}
template <int CH>
__host__ __device__ constexpr size_t shared_bytes(int np) { return region_bytes<CH>(np) + sizeof(Ctl); }

// f(i, j, row, column) over the thread's element pairs (row, column), (row,
// column + 1) of strip st of a matrix of nct column tiles.
template <class F>
__device__ __forceinline__ void each(const Geo& G, int st, int nct, F&& f) {
#pragma unroll
  for (int j = 0; j < kTC; ++j) {
    if (kTC * st + j < nct) {
#pragma unroll
      for (int i = 0; i < 2; ++i) f(i, j, G.r0 + 8 * i, kStrip * st + 8 * j + 2 * G.t);
    }
  }
}
// Such a pair of a workspace matrix (32-byte aligned: one access of a whole
// sector instead of two of half a sector each).
struct Pair {
  double2 v[2];
};
__device__ __forceinline__ Pair load2(const double2* p) {
  Pair x;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(x.v[0].x), "=d"(x.v[0].y), "=d"(x.v[1].x), "=d"(x.v[1].y)
               : "l"(p)
               : "memory");
  return x;
}
__device__ __forceinline__ void store2(double2* p, const Pair& x) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x.v[0].x), "d"(x.v[0].y), "d"(x.v[1].x),
               "d"(x.v[1].y)
               : "memory");
}

// Fragment at row r0 and chunk-relative k of a left factor in shared memory, rows
// of 8 with the place in the row XORed by swz(row).
__device__ __forceinline__ AFrag left_frag(const double2* S, int r, int t) {
  AFrag f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double2 v = S[r * 8 + ((t + 4 * h) ^ swz(r))];
    f.re[h] = v.x;
    f.im[h] = v.y;
  }
  return f;
}
// Fragment of column tile j of 8 rows of a strip in shared memory.
__device__ __forceinline__ AFrag right_frag(const double2* S, int j, const Geo& G) {
  AFrag f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = G.t + 4 * h;
    const double2 v = S[k * kStrip + 8 * j + (G.g ^ swz(k))];
    f.re[h] = v.x;
    f.im[h] = v.y;
  }
  return f;
}

// op(A) op(B) over kch chunks of 8, nct column tiles; f(row, column, pair) takes
// the elements, two neighbours at a time.  A, B: stored rows x cols elements, row stride ld,
// zero outside.  Both operands come through a ring of chunks in shared memory,
// four ahead: at one block per SM the blocks' matrices exceed L2, and fragments
// loaded from global memory one chunk ahead left the FP64 pipe 44 % idle at
// n = 192 (latency, passed on by the barriers).  Starts with a block barrier (the
// operands are then complete, the ring is free).
template <int CH, bool AC, bool BC, class F>
__device__ __forceinline__ void prod(const Left& A, const Left& B, int kch, int nct, double2* ring, const Geo& G,
                                     F&& f) {
  const int nst = (nct + kTC - 1) / kTC, as = 8 * G.NP, chunk_elems = as + 8 * kStrip;
  // A warp copies its own rows of A (lane: 4 elements of a chunk) and every
  // G.nthr / 32-th row of B's chunk (lane: a column).
  const int ar = G.r0 - G.g + (AC ? G.lane & 7 : G.lane >> 3), ak = AC ? G.lane >> 3 : G.lane & 7;
  const double2* const a0 = A.p + (AC ? ak * A.ld + ar : ar * A.ld + ak);
  const int ad = ar * 8 + (ak ^ swz(ar));
  int pst = 0, pkc = 0, ps = 0;  // next strip, chunk and ring slot to fetch
  auto copy = [](uint32_t dst, const double2* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
  };
  const uint32_t ring32 = umma::smem_u32(ring);
  auto fetch = [&] {
    if (pst < nst) {
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        if (CH > 1 && pkc + u >= kch) break;
        const uint32_t S = ring32 + (ps * CH + u) * chunk_elems * 16;
        const int kc = (pkc + u) * 8;
        if (G.active) {
          const double2* src = a0 + kc * (AC ? A.ld : 1);
          const int k = kc + ak;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // AC: rows + 8 (i & 1), k + 4 (i >> 1); else rows + 4 i (swz(r + 4) = swz(r) ^ 1)
            const int dr = AC ? 8 * (i & 1) : 4 * i, dk = AC ? 4 * (i >> 1) : 0;
            const bool in = AC ? (k + dk < A.rows && ar + dr < A.cols) : (ar + dr < A.rows && k < A.cols);
            const int d = AC ? ad + 64 * (i & 1) : ad + 32 * i;
            copy(S + 16 * (AC ? d ^ dk : d ^ (i & 1)), in ? src + (AC ? dk * A.ld + dr : dr * A.ld) : A.p, in);
          }
        }
        for (int x = G.warp; x < 8; x += G.nthr >> 5) {
          const int k = kc + x, c = pst * kStrip + G.lane;
          const bool in = BC ? (c < B.rows && k < B.cols) : (k < B.rows && c < B.cols);
          copy(S + 16 * (as + x * kStrip + (G.lane ^ swz(x))), in ? B.p + (BC ? c * B.ld + k : k * B.ld + c) : B.p, in);
        }
      }
      pkc += CH;
      if (pkc >= kch) {
        pkc = 0;
        ++pst;
      }
    }
    ps = ps + 1 == kRing<CH> ? 0 : ps + 1;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __syncthreads();
  for (int s = 0; s < kRing<CH> - 1; ++s) fetch();
  int slot = 0;
  // The warps of a scheduler fetch at different places among their MMAs, so that
  // one's address arithmetic runs under the others' MMAs.
  const int fpos = (G.warp >> 2 & 3) * CH;
#pragma unroll 1
  for (int st = 0; st < nst; ++st) {
    Acc c;
    c.zero();
#pragma unroll 1
    for (int k0 = 0; k0 < kch; k0 += CH) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kRing<CH> - 2) : "memory");
      __syncthreads();
      const double2* S = ring + slot * CH * chunk_elems;
      slot = slot + 1 == kRing<CH> ? 0 : slot + 1;
      if (!G.active) {
        fetch();
        continue;
      }
#pragma unroll
      for (int u = 0; u < CH; ++u, S += chunk_elems) {
        const bool live = CH == 1 || k0 + u < kch;
        AFrag a[2] = {left_frag(S, G.r0, G.t), left_frag(S, G.r0 + 8, G.t)};
        if (AC) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) a[i].im[h] = -a[i].im[h];
        }
#pragma unroll
        for (int j = 0; j < kTC; ++j) {
          if (kTC * u + j == fpos) fetch();
          if (live && kTC * st + j < nct) {
            AFrag b = right_frag(S + as, j, G);
            if (BC) {
              b.im[0] = -b.im[0];
              b.im[1] = -b.im[1];
            }
            chunk(c.re[0][j], c.im[0][j], a[0], b);
            chunk(c.re[1][j], c.im[1][j], a[1], b);
          }
        }
      }
    }
    if (G.active)
      each(G, st, nct, [&](int i, int j, int r, int cc) { f(r, cc, Pair{{c.get(i, j, 0), c.get(i, j, 1)}}); });
  }
}

// ------------------------------------------------------------ Gauss-Jordan --
// Inverse of the n x n matrix M (identity in the padding; M is used up), row
// stride NP, into out.  smem::gj_invert (see there for the algorithm and the
// pivot rule) on strips: the rows of M never move, the panel's positions are
// tracked per row.  A strip of 32 columns is factored in registers, four panels
// of 8, their left factors kept in shared memory; then every other strip is read
// once, takes the four updates in order and is written back, by the last pass at
// the final row and column.  The rows that the four updates multiply are the
// strip's 32 pivot rows, each as the updates before its own leave it: four warps
// work them out for the next strip (a column tile each) while the block updates
// this one, which leaves one barrier per strip.  Only the warps with rows take
// part (named barrier 1).
// sh.fail holds the status afterwards; the caller's block barrier publishes it
// and out.
__device__ __forceinline__ void gj_invert(double2* M, double2* out, int n, const Geo& G, unsigned char* region, Ctl& sh) {
  const int NP = G.NP, nt = 2 * NP, tid = G.tid, lane = G.lane, PE = NP * PS;
  const int nwa = NP >> 4;
  double2* const P = reinterpret_cast<double2*>(region);
  double2* const AS = P + pair_elems(NP);
  double2* const Bp = AS + 32 * NP;
  auto bar = [&] { asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory"); };
  const int pr_own = tid >> 1, cl = tid & 1, prow = pr_own * PS;
  const int nct = (n + 7) >> 3, nst = (nct + kTC - 1) / kTC;
  int pos[2] = {G.r0, G.r0 + 8};
  int cm = tid;  // threads 0 .. NP - 1: t_k(...t_0(tid)) over the interchanges done so far
#pragma unroll 1
  for (int sp = 0; sp < nst; ++sp) {
    Acc m;
    auto load = [&](int st) {
      m.zero();
      each(G, st, nct, [&](int i, int j, int r, int c) {
        const Pair x = load2(M + r * NP + c);
        m.set(i, j, 0, x.v[0]);
        m.set(i, j, 1, x.v[1]);
      });
    };
    load(sp);
    const int jn = min(kTC, nct - kTC * sp);
    unsigned piv = 0u;  // for panel s and row i: the row's place among the panel's pivots, 15 if none
    bar();  // the strips before have read their pivot rows (in P)
#pragma unroll 1
    for (int s = 0; s < jn; ++s) {
      const int k0 = kStrip * sp + 8 * s, jmax = min(8, n - k0);
      double2* const P0 = P;
      double2* const P1 = P + PE;
      unsigned key0 = 0u;
#pragma unroll
      for (int j = 0; j < kTC; ++j)
        if (j == s) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            double2* row = P0 + pos[i] * PS + 2 * G.t;
            row[0] = m.get(i, j, 0);
            row[1] = m.get(i, j, 1);
            if (G.t == 0 && pos[i] >= k0 && pos[i] < n) key0 = max(key0, smem::pivot_key<8>(m.get(i, j, 0), pos[i]));
          }
        }
      key0 = __reduce_max_sync(0xffffffffu, key0);
      if (lane == 0) sh.key[0][G.warp] = key0;
      if (tid == 0) sh.lam[0] = make_double2(1.0, 0.0);
      bar();
      double2 av[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) av[q] = P0[prow + cl + 2 * q];
      bool cand = pr_own >= k0 && pr_own < n;
      int fail = kOk;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= jmax) break;
        const double2* Pc = (j & 1) ? P1 : P0;
        double2* Pn = (j & 1) ? P0 : P1;
        const double2 fv = Pc[prow + j];
        const double2 lam = sh.lam[j & 1];
        const unsigned key = __reduce_max_sync(0xffffffffu, lane < nwa ? sh.key[j][lane] : 0u);
        const bool stop = key - 256u >= 0x7ff00000u - 256u;
        const int pr = min((int)(255u - (key & 255u)), NP - 1);
        const int ex = (int)(key >> 20);
        const double sc = (ex != 0 && ex < 2046) ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
        const double2* prow_p = Pc + pr * PS;
        const double2 pv = prow_p[j];
        const double2 ps = make_double2(pv.x * sc, pv.y * sc);
        double2 mv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) mv[q] = prow_p[cl + 2 * q];
        const bool isp = pr_own == pr;
        cand = cand && !isp;
        const double2 bb = isp ? lam : fv;
        const double nsc = isp ? sc : -sc;
        const double2 nb = make_double2(bb.x * nsc, bb.y * nsc);
        const double2 pe = isp ? make_double2(0.0, 0.0) : ps;
        unsigned nk = 0u;
#pragma unroll
        for (int qq = 0; qq < 4; ++qq) {
          const int q = (qq + (j + 1) / 2) % 4;  // the next pivot column first
          const int c = cl + 2 * q;
          const bool pivcol = q == j / 2 && cl == j % 2;
          const double2 mq = pivcol ? lam : mv[q];
          double2 v = make_double2(fma(nb.x, mq.x, -nb.y * mq.y), fma(nb.x, mq.y, nb.y * mq.x));
          cfma(v, pivcol ? make_double2(0.0, 0.0) : pe, av[q]);
          Pn[prow + c] = v;
          av[q] = v;
          if (j + 1 < 8 && qq == 0) {
            if (cl == (j + 1) % 2 && cand) nk = smem::pivot_key<8>(v, pr_own);
            nk = __reduce_max_sync(0xffffffffu, nk);
          }
        }
        if (j + 1 < 8 && lane == 0) sh.key[j + 1][G.warp] = nk;
        if (G.warp == nwa - 1 && lane == 0) {
          sh.lam[(j + 1) & 1] = cmul(lam, ps);
          sh.pivot[j] = pr;
        }
        if (stop) fail = fail ? fail : (key <= 255u ? kSingular : kNonFinite);
        if (j + 1 < jmax) bar();
      }
      if (G.warp == nwa - 1 && lane == 0) sh.fail = fail;
      bar();
      if (sh.fail) return;
      // Step j exchanged positions k0 + j and bl_j, where its pivot row stood by then.
      int np[2] = {pos[0], pos[1]}, bl[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j < jmax) {
          const int pr = sh.pivot[j], k = k0 + j;
          bl[j] = pr;
#pragma unroll
          for (int i = 0; i < j; ++i) bl[j] = bl[j] == k0 + i ? bl[i] : bl[j];
#pragma unroll
          for (int i = 0; i < 2; ++i) np[i] = np[i] == k ? bl[j] : (np[i] == bl[j] ? k : np[i]);
          cm = cm == k ? bl[j] : (cm == bl[j] ? k : cm);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const unsigned x = (unsigned)(np[i] - k0);
        piv |= (x < (unsigned)jmax ? x : 15u) << (8 * s + 4 * i);
        if (x < (unsigned)jmax) {
          if (G.t == 0) sh.prow[8 * s + x] = G.r0 + 8 * i;
#pragma unroll
          for (int j = 0; j < kTC; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              Bp[x * kStrip + 8 * j + ((2 * G.t + q) ^ swz(x))] = m.get(i, j, q);
              m.set(i, j, q, make_double2(0.0, 0.0));
            }
        }
      }
      const double2* Pf = (jmax & 1) ? P1 : P0;
      const double2 il = crecip_smith(sh.lam[jmax & 1]);
      AFrag a[2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double2 v = cmul(Pf[pos[i] * PS + G.t + 4 * h], il);
          a[i].re[h] = v.x;
          a[i].im[h] = v.y;
          AS[(s * NP + G.r0 + 8 * i) * 8 + ((G.t + 4 * h) ^ swz(G.g))] = v;
        }
      bar();
#pragma unroll
      for (int j = 0; j < kTC; ++j) {
        if (j == s) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) m.set(i, j, q, cmul(Pf[pos[i] * PS + 2 * G.t + q], il));
        } else if (j < jn) {
          AFrag b;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int kk = G.t + 4 * h;
            const double2 v = Bp[kk * kStrip + 8 * j + (G.g ^ swz(kk))];
            b.re[h] = kk < jmax ? v.x : 0.0;
            b.im[h] = kk < jmax ? v.y : 0.0;
          }
          chunk(m.re[0][j], m.im[0][j], a[0], b);
          chunk(m.re[1][j], m.im[1][j], a[1], b);
        }
      }
      pos[0] = np[0];
      pos[1] = np[1];
      bar();  // the panel and its pivot rows are read
    }
    const bool last = sp == nst - 1;
    if (last) {
      if (tid < NP) sh.cinv[cm] = tid;
      bar();
    }
    auto put = [&](int st) {
      each(G, st, nct, [&](int i, int j, int r, int c) {
        if (last) {
          out[pos[i] * NP + sh.cinv[c]] = m.get(i, j, 0);
          out[pos[i] * NP + sh.cinv[c + 1]] = m.get(i, j, 1);
        } else {
          store2(M + r * NP + c, Pair{{m.get(i, j, 0), m.get(i, j, 1)}});
        }
      });
    };
    put(sp);
    // ---- the other strips ----
    const int jlast = min(8, n - (kStrip * sp + 8 * (jn - 1)));  // pivots of the last panel
    // T <- the pivot rows of strip st, each panel's as the updates before it leave them
    auto pivot_rows = [&](int st, double2* T) {
      for (int j = G.warp; j < kTC; j += nwa) {
        if (kTC * st + j >= nct) break;
        double re[kTC][2], im[kTC][2];
        int row[kTC];
#pragma unroll
        for (int s = 0; s < kTC; ++s) {
          row[s] = s < jn && G.g < (s == jn - 1 ? jlast : 8) ? sh.prow[8 * s + G.g] : -1;
#pragma unroll
          for (int q = 0; q < 2; ++q) re[s][q] = im[s][q] = 0.0;
          if (row[s] >= 0) {
            const Pair x = load2(M + row[s] * NP + kStrip * st + 8 * j + 2 * G.t);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              re[s][q] = x.v[q].x;
              im[s][q] = x.v[q].y;
            }
          }
        }
#pragma unroll
        for (int s = 0; s < kTC; ++s) {
          if (s >= jn) break;
#pragma unroll
          for (int q = 0; q < 2; ++q)
            T[(8 * s + G.g) * kStrip + 8 * j + ((2 * G.t + q) ^ swz(G.g))] =
                row[s] >= 0 ? make_double2(re[s][q], im[s][q]) : make_double2(0.0, 0.0);
          __syncwarp();
          const AFrag b = right_frag(T + 8 * s * kStrip, j, G);
#pragma unroll
          for (int s2 = s + 1; s2 < kTC; ++s2)
            if (s2 < jn) chunk(re[s2], im[s2], left_frag(AS + s * NP * 8, max(row[s2], 0), G.t), b);
        }
      }
    };
    const int first = sp == 0 ? 1 : 0;
    if (first < nst) pivot_rows(first, P);
    bar();
    int par = 0;
#pragma unroll 1
    for (int st = first; st < nst; par ^= 1) {
      const int nx = st + 1 == sp ? st + 2 : st + 1;
      load(st);
      if (nx < nst) pivot_rows(nx, P + (par ^ 1) * kStrip * kStrip);
      const double2* T = P + par * kStrip * kStrip;
#pragma unroll 1
      for (int s = 0; s < jn; ++s, T += 8 * kStrip) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if ((piv >> (8 * s + 4 * i) & 15u) < 8u) {
#pragma unroll
            for (int j = 0; j < kTC; ++j)
#pragma unroll
              for (int q = 0; q < 2; ++q) m.set(i, j, q, make_double2(0.0, 0.0));
          }
        const AFrag a[2] = {left_frag(AS + s * NP * 8, G.r0, G.t), left_frag(AS + s * NP * 8, G.r0 + 8, G.t)};
#pragma unroll
        for (int j = 0; j < kTC; ++j) {
          if (kTC * st + j < nct) {
            const AFrag b = right_frag(T, j, G);
            chunk(m.re[0][j], m.im[0][j], a[0], b);
            chunk(m.re[1][j], m.im[1][j], a[1], b);
          }
        }
      }
      put(st);
      st = nx;
      bar();  // the next strip's pivot rows are there, this one's are read
    }
  }
}

// ------------------------------------------------------------ Sancho-Rubio --
// Decimation of one point (recurrence, stopping rule and final g of
// smem::sr_f64_kernel).  W: 7 NP^2 of workspace.  Returns the status, *iters
// the sweeps; *g the padded surface GF (row stride NP) when kOk.
template <int CH>
__device__ __forceinline__ int sr_point(int n, const Geo& G, const double2* h00, const double2* h01, const double2* h10,
                                        double2 z, double tol, int maxiter, double2* W, unsigned char* region, Ctl& sh,
                                        int* iters, double2** g) {
  const int NP = G.NP, kch = (n + 7) >> 3, nct = kch, nst = (nct + kTC - 1) / kTC;
  const int M2 = NP * NP;
  double2 *al = W, *be = W + M2, *m = W + 4 * M2, *gi = W + 5 * M2, *bg = W + 6 * M2;
  double2 *const ep = W + 2 * M2, *const es = W + 3 * M2;
  double2* const ring = reinterpret_cast<double2*>(region);
  auto left = [&](const double2* p) { return Left{p, NP, NP, NP}; };
  if (G.active)
    for (int st = 0; st < nst; ++st)
      each(G, st, nct, [&](int, int, int r, int c0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int c = c0 + q, e = r * NP + c;
          const bool in = r < n && c < n;
          const double2 e0 = in ? h00[r * n + c] : make_double2(0.0, 0.0);
          ep[e] = e0;
          es[e] = e0;
          al[e] = in ? h01[r * n + c] : make_double2(0.0, 0.0);
          be[e] = in ? (h10 ? h10[r * n + c] : cconj(h01[c * n + r])) : make_double2(0.0, 0.0);
        }
      });
  const double tol2 = tol * tol;
  int status = kOk, it = 0;
  bool converged = false;
  for (;;) {
    if (!converged) ++it;
    if (G.active) {
      const double2* src = converged ? es : ep;
      for (int st = 0; st < nst; ++st)
        each(G, st, nct, [&](int, int, int r, int c0) {
          Pair x = load2(src + r * NP + c0);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int c = c0 + q;
            if (r < n && c < n) x.v[q] = r == c ? csub(z, x.v[q]) : cneg(x.v[q]);
            else x.v[q] = make_double2(r == c ? 1.0 : 0.0, 0.0);
          }
          store2(m + r * NP + c0, x);
        });
    }
    __syncthreads();
    if (G.active) gj_invert(m, gi, n, G, region, sh);
    __syncthreads();
    status = sh.fail;
    if (status != kOk || converged) break;
    double2* const ag = m;
    auto to = [&](double2* dst) { return [=](int r, int c, const Pair& v) { store2(dst + r * NP + c, v); }; };
    prod<CH, false, false>(left(al), left(gi), kch, nct, ring, G, to(ag));
    prod<CH, false, false>(left(be), left(gi), kch, nct, ring, G, to(bg));
    int bad = 0;
    double e2 = 0.0;
    auto add = [&](double2* dst, const Pair& v) {
      Pair x = load2(dst);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        x.v[q] = cadd(x.v[q], v.v[q]);
        bad |= !cfinite(x.v[q]);
      }
      store2(dst, x);
    };
    auto next = [&](double2* dst, const Pair& v) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        bad |= !cfinite(v.v[q]);
        e2 = fmax(e2, cabs2(v.v[q]));
      }
      store2(dst, v);
    };
    prod<CH, false, false>(left(ag), left(be), kch, nct, ring, G, [&](int r, int c, const Pair& v) {
      add(es + r * NP + c, v);
      add(ep + r * NP + c, v);
    });
    prod<CH, false, false>(left(bg), left(be), kch, nct, ring, G, [&](int r, int c, const Pair& v) { next(gi + r * NP + c, v); });
    prod<CH, false, false>(left(bg), left(al), kch, nct, ring, G, [&](int r, int c, const Pair& v) { add(ep + r * NP + c, v); });
    // beta g is used up, and its rows belong to the warp that reads them
    prod<CH, false, false>(left(ag), left(al), kch, nct, ring, G, [&](int r, int c, const Pair& v) { next(bg + r * NP + c, v); });
    double2* const oa = al;
    double2* const ob = be;
    al = bg;
    be = gi;
    bg = oa;
    gi = ob;
    if (block_any(bad)) {
      status = sr_failure_status(it, n, h00, h01, h10, z);
      break;
    }
    converged = block_max(e2, sh.red) < tol2;
    if (!converged && it == maxiter) {
      status = kMaxIter;
      break;
    }
  }
  *iters = it;
  *g = gi;
  return status;
}

// ---------------------------------------------------------------- RGF sweep --
struct Point {
  int n, nl, nr, L;
  const double2* D;
  long long d_ls;
  const double2* C;
  long long c_ls;
  const double2 *VL, *VR, *gL, *gR;
  double2 z;
};
// Workspace of rgf_point: five NP^2 matrices, then Sigma_L and Sigma_R.
__host__ __device__ constexpr size_t rgf_elems(int np, int n) { return 5 * (size_t)np * np + 2 * (size_t)n * n; }

template <int CH>
__device__ __forceinline__ int rgf_point(const Point& q, const Geo& G, double2* W, unsigned char* region, Ctl& sh, double* t) {
  const int NP = G.NP, n = q.n, kch = (n + 7) >> 3, nct = kch, M2 = NP * NP;
  double2 *const gl = W, *const m = W + M2, *const w = W + 2 * M2, *const u = W + 3 * M2, *const g0 = W + 4 * M2;
  double2 *const sigL = W + 5 * M2, *const sigR = sigL + (long long)n * n;
  double2* const ring = reinterpret_cast<double2*>(region);
  auto left = [&](const double2* p) { return Left{p, NP, NP, NP}; };
  auto to = [&](double2* dst) { return [=](int r, int c, const Pair& v) { store2(dst + r * NP + c, v); }; };
  for (int side = 0; side < 2; ++side) {  // Sigma = V g V^H
    const int nl = side ? q.nr : q.nl, lch = (nl + 7) >> 3;
    const Left V{side ? q.VR : q.VL, nl, n, nl};
    double2* const S = side ? sigR : sigL;
    prod<CH, false, false>(V, Left{side ? q.gR : q.gL, nl, nl, nl}, lch, lch, ring, G, to(u));
    prod<CH, false, true>(left(u), V, lch, nct, ring, G, [=](int r, int c, const Pair& v) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (r < n && c + q < n) S[r * n + c + q] = v.v[q];
    });
  }
  int status = kOk;
  for (int l = 0; l < q.L; ++l) {
    const double2* D = q.D + (long long)l * q.d_ls;
    const double2* SR = l == q.L - 1 ? sigR : nullptr;
    // M = z - D_l - (C^H g C, or Sigma_L on layer 0) [- Sigma_R on the last layer]
    auto form = [&](int r, int c0, Pair x) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + h;
        double2 v = make_double2(r == c ? 1.0 : 0.0, 0.0);
        if (r < n && c < n) {
          v = csub(cneg(D[r * n + c]), x.v[h]);
          if (SR) v = csub(v, SR[r * n + c]);
          if (r == c) v = cadd(v, q.z);
        }
        x.v[h] = v;
      }
      store2(m + r * NP + c0, x);
    };
    auto part = [n](const double2* S, int r, int c) { return r < n && c < n ? S[r * n + c] : make_double2(0.0, 0.0); };
    if (l == 0) {
      __syncthreads();
      if (G.active)
        for (int st = 0; st * kTC < nct; ++st)
          each(G, st, nct, [&](int, int, int r, int c) { form(r, c, Pair{{part(sigL, r, c), part(sigL, r, c + 1)}}); });
    } else {
      const Left C{q.C + (long long)(l - 1) * q.c_ls, n, n, n};
      prod<CH, false, false>(left(g0), C, kch, nct, ring, G, to(u));  // U = G_{0,l-1} C
      prod<CH, false, false>(left(gl), C, kch, nct, ring, G, to(w));  // W = g_{l-1} C
      prod<CH, true, false>(C, left(w), kch, nct, ring, G, [&](int r, int c, const Pair& v) { form(r, c, v); });
    }
    __syncthreads();
    if (G.active) gj_invert(m, l == 0 ? g0 : gl, n, G, region, sh);
    __syncthreads();
    status = sh.fail;
    if (status != kOk) break;
    if (l == 0) {
      if (q.L > 1)
        for (int e = G.tid; e < M2; e += G.nthr) gl[e] = g0[e];
    } else {
      prod<CH, false, false>(left(u), left(gl), kch, nct, ring, G, to(g0));  // G_{0,l} = U g_l
    }
  }
  __syncthreads();
  double tval = 0.0;
  if (status == kOk) {
    // T = Re sum_ij (Gamma_L G Gamma_R)_ij conj(G)_ij
    if (G.active)
      for (int st = 0; st * kTC < nct; ++st)
        each(G, st, nct, [&](int, int, int r, int c) {
          store2(w + r * NP + c, Pair{{gamma_of(sigL, n, r, c), gamma_of(sigL, n, r, c + 1)}});
          store2(m + r * NP + c, Pair{{gamma_of(sigR, n, r, c), gamma_of(sigR, n, r, c + 1)}});
        });
    double* const terms = reinterpret_cast<double*>(gl);
    prod<CH, false, false>(left(w), left(g0), kch, nct, ring, G, to(u));
    prod<CH, false, false>(left(u), left(m), kch, nct, ring, G, [&](int r, int c, const Pair& v) {
      const Pair x = load2(g0 + r * NP + c);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double s = 0.0;
        s += v.v[h].x * x.v[h].x + v.v[h].y * x.v[h].y;
        terms[r * NP + c + h] = s;
      }
    });
    __syncthreads();
    // summed as in mid::trace_t
    const int np16 = (max(n, max(q.nl, q.nr)) + 15) >> 4;
    for (int v = G.warp; v < 8; v += G.nthr >> 5) {
      double s = 0.0;
      for (int b = v; b < np16 * np16; b += 8)
        for (int e = 0; e < 8; ++e) {
          const int r = (b / np16) * 16 + G.g + 8 * ((e >> 1) & 1), c = (b % np16) * 16 + 8 * (e >> 2) + 2 * G.t + (e & 1);
          if (r < NP && c < 8 * nct) s += terms[r * NP + c];
        }
      s = warp_sum(s);
      if (G.lane == 0) sh.red[v] = s;
    }
    __syncthreads();
    tval = warp_sum(G.lane < 8 ? sh.red[G.lane] : 0.0);
    if (!isfinite(tval)) status = kNonFinite;
    __syncthreads();
  }
  *t = tval;
  return status;
}

}  // namespace big
}  // namespace negf
