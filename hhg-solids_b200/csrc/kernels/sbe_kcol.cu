// Column-tile FP64 propagation for two orbitals with a Hermitian placement and a cell box symmetric about
// zero and at most 7 x 7 cells (the 2-orbital configurations).
//
// Same propagation as sbe_kcol_any.cu (the k-space-resident RK4 of src/solver.cpp:86-181 with the current of
// src/observable.cpp:16-30; KM: the k-space solver of src/solver_kspace.cpp).
//
// H = (D, o), D = H00 - H11, o = H01, is all the commutator needs:
//   k00 = 2 (o.y x.x - o.x x.y) = -k11,  k01 = -i (D x - d o),  x = X01, d = X00 - X11.
// With t = e^{-2 pi i m1 / N1} and G(-n1) = G(n1)^+ every part of H is T0 + sum_{n1 > 0} (Re t^n1 A(n1) + Im t^n1
// B(n1)), A and B the same for a whole k-grid column.  Rows m1 and m1 + N1/2 have t^n1 equal for even n1 and
// opposite for odd, so a thread takes both: the even and the odd half of the sum are formed once.  The same
// holds for the window's row twiddles in the current: it needs the sum of the pair's states for n1 = 0, +-2 and
// their difference for n1 = +-1.
//
// Column tables (column_tables): per k-grid column and step, with the field applied: real-space solver, H at t
// and t + dt (at t + dt/2 the field is their mean, so the middle stages run on the sum of the two with the factor
// in the stage's constants); k-space solver, H at t + dt/2 and t + dt; and the window coefficients.
//
// A CTA takes a tile of up to 32 pairs of one column for all steps of the launch (propagate_tile), a thread per
// pair, states in registers.  Every kIv steps it has staged kIv steps of states in shared memory; during the next
// kIv they are summed over the rows (five real sums per state value; lane = quarter of the rows, step, value pair;
// the twiddles in registers) and the sums contracted with the window coefficients.  Where the tiles are many one
// warp does both, without a barrier; where they are few a second warp takes the sums (SPLIT), and the two meet
// every kIv steps.  The other CTAs of a launch form the next launch's tables, so only a pulse's first ones are
// waited for.
//
// What bounds it: FP64 operations on three different operands take about 3.2 cycles of a sub-partition (register
// reads; 2.2 with shared operands), 172 of them per pair and step: 550 cycles a step for each tile of the
// sub-partition with the most tiles.  Where tiles are few most sub-partitions have none, and a tile's state warp is
// bound by the same: 144 such operations a step, 460 of the 504 cycles that a step of 60 x 60 takes.
//
// Measured on B200 (1965 MHz), 4096 steps, one field axis: 200 x 200 2.60 ms (one k-point per thread, window and
// Peierls factors summed per CTA: 4.36), k-space solver 2.49 ms (5.75); 60 x 60 1.05 ms (thread-per-k-point kernel
// with per-thread cell sums: 6.16).
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>

#include "sbe_device.h"
#include "smem_limit.h"

namespace hhg {
namespace {

constexpr int kIv = 4;          // steps per staged interval
constexpr int kKcolChunk = 256; // steps per launch
constexpr int kTabPts = 32;     // evaluation points of a table CTA

__device__ __forceinline__ double2 kc_mul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 kc_fma(double2 a, double2 b, double2 c) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
  return c;
}
__device__ __forceinline__ int kc_wrap(long long x, int n) {
  const int r = (int)(x % n);
  return r < 0 ? r + n : r;
}
__device__ __forceinline__ void kc_cp16(void* dst_smem, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// The column tables in global scratch, in doubles.  A table: T0 of (D, o.x, o.y, -), then per n1 = 1..Q the
// pairs (A, B) of each.  A step's record: real-space solver the tables at t and t + dt and the window
// coefficients [4 state values][nj][4 rows] complex; k-space solver the tables at t + dt/2 and t + dt, with the
// chunk's first table and the (constant) coefficients in a block per column after all records.
// (Room for kNj current axes: models in the plane have two.)
constexpr int kNj = 2;
template <int Q, bool KM>
struct Tables {
  static constexpr int TBL = 4 + 6 * Q;
  static constexpr int W2 = 2 * Q + 1;  // cells of a box row (narrower boxes padded with zeros)
  static constexpr int COEF = 32 * kNj, REC = 2 * TBL + (KM ? 0 : COEF), COL = KM ? TBL + COEF : 0;
};

// One warp: column m2, points l0 .. l0 + kTabPts - 1 of the steps [step0, step1).  Real-space solver: a point per
// step; k-space solver: points 2 step0 + 1, ... (two per step), and the first group's extra point 2 step0.
template <int Q, bool KM>
struct TabSmem {
  static constexpr int W2 = 2 * Q + 1, NP = kTabPts + (KM ? 1 : 0);
  double2 p2[NP][W2 + 4];       // column factors: box cells n2 = -Q..Q, window cells -2..1
  double2 p1[NP][Q + 5];        // row factors: n1 = 0..Q, window rows -2..1
  double2 xc[4][Q + 1][3][W2];  // X00 - X11, X01, X10
  double2 tw2[W2 + 4];
  double es[KM ? kTabPts / 2 + 1 : kTabPts][9];
};
template <int Q, bool KM>
__device__ __forceinline__ void column_tables(const SolveTables& t, const GroupTables& gt, int step0, int step1, int m2,
                                              int l0, int chunk, double* out, TabSmem<Q, KM>& S) {
  using TT = Tables<Q, KM>;
  constexpr int TBL = TT::TBL, W2 = TT::W2;
  const int lane = threadIdx.x & 31, nmat = 1 + t.nax, nj = t.nj;
  const int half = (t.b1n - 1) / 2, npw = 2 * t.np + 1;
  const int steps = step1 - step0, npts = KM ? 2 * steps : steps, ns = min(kTabPts, npts - l0);
  const int first = KM && l0 == 0 ? 1 : 0, np = ns + first;
  const double2 zero = make_double2(0.0, 0.0);
  // local point l: l < first: the chunk's first point; else point l0 + l - first
  auto row_of = [&](int l) { return KM ? (l < first ? 2 * step0 : 2 * step0 + 1 + l0 + l - first) : step0 + l0 + l; };
  // (the steps' field samples of the group)
  const int st0 = KM ? l0 >> 1 : l0, nst = KM ? (ns + 1) >> 1 : ns;
  for (int idx = lane; idx < nst * 9; idx += 32) S.es[idx / 9][idx % 9] = t.es[(size_t)(step0 + st0) * 9 + idx];
  if (lane < W2 + 4) S.tw2[lane] = t.T2[kc_wrap(m2 * (lane < W2 ? lane - Q : lane - W2 - 2), t.N2)];
  for (int idx = lane; idx < nmat * (Q + 1) * W2; idx += 32) {
    const int n2 = idx % W2 - Q, q = (idx / W2) % (Q + 1), mat = idx / (W2 * (Q + 1));
    const bool on = q <= half && n2 >= t.b2lo && n2 <= -t.b2lo;
    const double2* x = gt.Xbox64 + (on ? ((size_t)(mat * t.b1n + half + q) * t.b2n + n2 - t.b2lo) * 4 : 0);
    const double2 x0 = x[0], x1 = x[1], x2 = x[2], x3 = x[3];
    S.xc[mat][q][0][n2 + Q] = on ? make_double2(x0.x - x3.x, x0.y - x3.y) : zero;
    S.xc[mat][q][1][n2 + Q] = on ? x1 : zero;
    S.xc[mat][q][2][n2 + Q] = on ? x2 : zero;
  }
  const int clampq = min(Q, t.np);
  for (int idx = lane; idx < np * (Q + 5); idx += 32) {
    const int l = idx / (Q + 5), q = idx % (Q + 5);
    const double2* P = gt.P64 + (size_t)row_of(l) * 2 * npw + t.np;
    S.p1[l][q] = q <= Q ? P[min(q, clampq)] : P[q - Q - 3];
  }
  __syncwarp();
  for (int idx = lane; idx < np * (W2 + 4); idx += 32) {
    const int l = idx / (W2 + 4), q = idx % (W2 + 4), n2 = q < W2 ? q - Q : q - W2 - 2;
    const double2* P = gt.P64 + (size_t)row_of(l) * 2 * npw + npw + t.np;
    S.p2[l][q] = (KM && q >= W2) ? S.tw2[q] : kc_mul(S.tw2[q], P[max(-clampq, min(clampq, n2))]);
  }
  __syncwarp();
  double* base = out + (size_t)m2 * chunk * TT::REC;
  double* colb = out + (size_t)t.N2 * chunk * TT::REC + (size_t)m2 * TT::COL;
  // Items (point, row n1, D or o).
  for (int idx = lane; idx < np * (Q + 1) * 2; idx += 32) {
    const int l = idx % np, qk = idx / np, q = qk >> 1, kind = qk & 1;
    const int pt = l0 + l - first;  // point in the chunk; its step and field samples
    const int st = KM ? pt >> 1 : pt;
    const double* es = S.es[l < first ? 0 : st - st0];
    const int e0 = KM ? (l < first ? 0 : ((pt & 1) ? 6 : 3)) : 0, e1 = 6;
    double2 a0 = zero, a1 = zero, b0 = zero, b1 = zero;  // first and second sample: D or G01, and G10
    for (int mat = 0; mat < nmat; ++mat) {
      const int ax = mat == 0 ? 0 : (mat == 1 ? t.ax_id[0] : (mat == 2 ? t.ax_id[1] : t.ax_id[2]));
      const double f0 = mat ? es[e0 + ax] : 1.0, f1 = mat ? es[e1 + ax] : 1.0;
      double2 u = zero, h = zero;
#pragma unroll
      for (int n = 0; n < W2; ++n) {
        u = kc_fma(S.p2[l][n], S.xc[mat][q][kind][n], u);
        if (kind) h = kc_fma(S.p2[l][n], S.xc[mat][q][2][n], h);
      }
      u = kc_mul(S.p1[l][q], u);
      h = kc_mul(S.p1[l][q], h);
      a0 = make_double2(fma(f0, u.x, a0.x), fma(f0, u.y, a0.y));
      b0 = make_double2(fma(f0, h.x, b0.x), fma(f0, h.y, b0.y));
      a1 = make_double2(fma(f1, u.x, a1.x), fma(f1, u.y, a1.y));
      b1 = make_double2(fma(f1, h.x, b1.x), fma(f1, h.y, b1.y));
    }
#pragma unroll
    for (int f = 0; f < (KM ? 1 : 2); ++f) {
      const double2 a = f ? a1 : a0, b = f ? b1 : b0;
      double* d = l < first ? colb : base + (size_t)st * TT::REC + (KM ? (pt & 1) : f) * TBL;
      if (q == 0) {
        if (kind == 0)
          d[0] = a.x;
        else
          d[1] = a.x, d[2] = a.y;
      } else {
        double2* dq = reinterpret_cast<double2*>(d + 4 + 6 * (q - 1));
        if (kind == 0) {
          dq[0] = make_double2(2.0 * a.x, -2.0 * a.y);
        } else {  // S = G01 + conj G10, D = G01 - conj G10
          dq[1] = make_double2(a.x + b.x, -(a.y + b.y));
          dq[2] = make_double2(a.y - b.y, a.x - b.x);
        }
      }
    }
  }
  // Window coefficients [value][axis][row] of rho00, rho11, Re rho01 (V01 + V10) and Im rho01 (-i (V01 - V10)), a lane
  // each.
  const int per = 16 * nj;
  const int nwp = KM ? first : ns;
  for (int c = lane; c < per; c += 32) {
    const int w1 = c & 3, a = (c >> 2) % nj, vv = (c >> 2) / nj;
    double2 vc[4];
#pragma unroll
    for (int w2 = 0; w2 < 4; ++w2) {
      const double2* x = gt.Xwin64 + (size_t)(a * 4 + w1) * 16 + 4 * w2;
      const double2 x0 = x[0], x1 = x[1], x2 = x[2], x3 = x[3];
      vc[w2] = vv == 0   ? x0
               : vv == 1 ? x3
               : vv == 2 ? make_double2(x1.x + x2.x, x1.y + x2.y)
                         : make_double2(x1.y - x2.y, x2.x - x1.x);
    }
#pragma unroll 2
    for (int l = 0; l < nwp; ++l) {
      double2 acc = zero;
#pragma unroll
      for (int w2 = 0; w2 < 4; ++w2) acc = kc_fma(S.p2[l][W2 + w2], vc[w2], acc);
      if (!KM) acc = kc_mul(S.p1[l][Q + 1 + w1], acc);
      double* d = KM ? colb + TBL : base + (size_t)(l0 + l) * TT::REC + 2 * TBL;
      reinterpret_cast<double2*>(d)[c] = acc;
    }
  }
}

template <int Q, bool KM>
struct PropSmem {
  using TT = Tables<Q, KM>;
  static constexpr int YS = 34;  // row stride of the staged states, 2 mod 16 doubles: the eight rows of one load
                                 // phase fall in distinct banks
  double rb[3][kIv][TT::REC];    // records: the previous interval's (coefficients), this one's, the next one's
  double cb[KM ? TT::COL : 2];   // the column's block
  double y[2][4][2 * kIv][YS];   // row class 2 (value & 1) + (difference), row 2 step + value / 2
};

struct KcolArgs {
  SolveTables t;      // steps [step0, step1) to propagate
  GroupTables gt;
  const double* cur;  // their tables
  double* next;       // tables of [next0, next1), formed by the CTAs from nprop on
  int next0, next1, chunk, R, vctas, nprop;
  double2 *rho, *Jpart;
};

// SPLIT: warp 0 propagates, warp 1 forms the current; otherwise one warp does both.
template <int Q, bool KM, bool SPLIT>
__device__ __forceinline__ void propagate_tile(const KcolArgs& A, int v, int tile, PropSmem<Q, KM>& S) {
  using TT = Tables<Q, KM>;
  constexpr int TBL = TT::TBL;
  const SolveTables& t = A.t;
  const int lane = threadIdx.x & 31, nj = t.nj, hN = t.N1 / 2;
  const bool steps = !SPLIT || threadIdx.x < 32, sums = !SPLIT || threadIdx.x >= 32;
  auto sync = [] {
    if (SPLIT)
      __syncthreads();
    else
      __syncwarp();
  };
  const int step0 = t.step0, step1 = t.step1, nint = (step1 - step0 + kIv - 1) / kIv;
  const double dt = t.dt, prefac = 0.1666666666666 * dt;
  const int pairs = min(t.row1 - t.row0, hN), tpc = (pairs + A.R - 1) / A.R;
  const int m2 = tile / tpc, i0 = (tile % tpc) * A.R, m10 = t.row0 + i0;
  const int nown = min(A.R, pairs - i0);

  const double* recs = A.cur + (size_t)m2 * A.chunk * TT::REC;
  auto fetch = [&](int iv) {  // records of interval iv into buffer iv % 3
    const int n = min(kIv, step1 - step0 - iv * kIv) * TT::REC / 2;
    double* dst = &S.rb[iv % 3][0][0];
    const double* src = recs + (size_t)iv * kIv * TT::REC;
    if (n == kIv * TT::REC / 2) {
#pragma unroll
      for (int q = 0; q < (kIv * TT::REC / 2 + 31) / 32; ++q)
        if (q * 32 + lane < kIv * TT::REC / 2) kc_cp16(dst + 2 * (q * 32 + lane), src + 2 * (q * 32 + lane));
    } else {
      for (int idx = lane; idx < n; idx += 32) kc_cp16(dst + 2 * idx, src + 2 * idx);
    }
  };
  sync();  // the previous tile's readers are done
  if (sums) fetch(0);
  if (KM && sums) {
    const double* src = A.cur + (size_t)t.N2 * A.chunk * TT::REC + (size_t)m2 * TT::COL;
    for (int idx = lane; idx < TT::COL / 2; idx += 32) kc_cp16(S.cb + 2 * idx, src + 2 * idx);
  }
  if (sums)
    for (int idx = lane; idx < 4 * 2 * kIv * S.YS; idx += 32) (&S.y[1][0][0][0])[idx] = 0.0;  // "interval -1"

  // Sums over the rows: lane = (quarter kq of the rows, step, value pair); its rows' twiddles.
  const int kq = lane >> 3, sl = lane & 7;
  double twr[8][4];  // cos, sin, cos 2, sin 2 of 2 pi m1 / N1
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m1 = min(m10 + kq * 8 + i, t.N1 - 1);
    const double2 a = t.T1[m1], b = t.T1[2 * m1 < t.N1 ? 2 * m1 : 2 * m1 - t.N1];
    twr[i][0] = a.x;
    twr[i][1] = -a.y;
    twr[i][2] = b.x;
    twr[i][3] = -b.y;
  }
  // The lane's place in the contraction: value vv, axis ja, step sl / 2.
  const bool hi = lane >= 16;
  const int ja = kq & 1, jcoef = ((2 * (lane & 1) + (hi ? 1 : 0)) * nj + ja) * 4;
  double2* Jrow = A.Jpart + ((size_t)v * t.nt + step0 + (sl >> 1)) * 3 + (ja ? t.j_id[1] : t.j_id[0]);
  double z[2][5];
  auto clear = [&] {
#pragma unroll
    for (int i = 0; i < 5; ++i) z[0][i] = z[1][i] = 0.0;
  };
  // Rows 2 part, 2 part + 1 of the quarter, staged in buffer b.
  auto sum_part = [&](int part, int b) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double2 yp = *reinterpret_cast<const double2*>(&S.y[b][2 * u][sl][kq * 8 + 2 * part]);
      const double2 ym = *reinterpret_cast<const double2*>(&S.y[b][2 * u + 1][sl][kq * 8 + 2 * part]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double* w = twr[2 * part + e];
        const double p = e ? yp.y : yp.x, m = e ? ym.y : ym.x;
        z[u][0] += p;
        z[u][1] = fma(w[0], m, z[u][1]);
        z[u][2] = fma(w[1], m, z[u][2]);
        z[u][3] = fma(w[2], p, z[u][3]);
        z[u][4] = fma(w[3], p, z[u][4]);
      }
    }
  };
  // Interval iv's sums over the quarters (the upper lanes keep the second value's, the lower the first's), times
  // the coefficients, into its row of partials; iv < 0: nothing is stored.
  auto finish = [&](int iv) {
    double q[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const double keep = hi ? z[1][i] : z[0][i], send = hi ? z[0][i] : z[1][i];
      q[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      q[i] += __shfl_xor_sync(0xffffffffu, q[i], 8);
    }
    const bool on = iv >= 0 && ja < nj && step0 + iv * kIv + (sl >> 1) < step1;
    double re = 0.0, im = 0.0;
    if (on) {
      // rows n1 = -2, -1, 0, 1 have the sums (q3, q4), (q1, q2), (q0, 0), (q1, -q2)
      const double2* cf = reinterpret_cast<const double2*>(KM ? S.cb + TBL : &S.rb[iv % 3][sl >> 1][2 * TBL]) + jcoef;
      const double2 f0 = cf[0], f1 = cf[1], f2 = cf[2], f3 = cf[3];
      re = fma(f0.x, q[3], fma(-f0.y, q[4], fma(f1.x + f3.x, q[1], fma(f3.y - f1.y, q[2], f2.x * q[0]))));
      im = fma(f0.x, q[4], fma(f0.y, q[3], fma(f1.x - f3.x, q[2], fma(f1.y + f3.y, q[1], f2.y * q[0]))));
    }
    re += __shfl_xor_sync(0xffffffffu, re, 1);
    im += __shfl_xor_sync(0xffffffffu, im, 1);
    re += __shfl_xor_sync(0xffffffffu, re, 16);
    im += __shfl_xor_sync(0xffffffffu, im, 16);
    if (on && (lane & 17) == 0) {
      double2* dst = Jrow + (ptrdiff_t)iv * kIv * 3;
      // the virtual CTA's first tile writes its row (cleared before the launch) without reading it
      const double2 old = tile == v ? make_double2(0.0, 0.0) : *dst;
      *dst = make_double2(old.x + re, old.y + im);
    }
  };

  // States of the k-points (m1, m2) and (m1 + N1/2, m2), m1 = m10 + lane.
  const bool on0 = steps && lane < nown, on1 = on0 && m10 + lane + hN < t.row1;
  const size_t k0 = (size_t)(m10 + (on0 ? lane : 0)) * t.N2 + m2, k1 = on1 ? k0 + (size_t)hN * t.N2 : k0;
  double r00[2] = {}, r11[2] = {}, ux[2] = {}, uy[2] = {}, twa[Q], twb[Q];
  double hD[2] = {}, hx[2] = {}, hy[2] = {};  // k-space solver: H at the step's t, carried
  auto get = [&](size_t k, int j) {
    r00[j] = A.rho[k * 4].x;
    r11[j] = A.rho[k * 4 + 3].x;
    ux[j] = A.rho[k * 4 + 1].x;
    uy[j] = A.rho[k * 4 + 1].y;
  };
  if (on0) get(k0, 0);
  if (on1) get(k1, 1);
  {
    const int m1 = min(m10 + lane, t.N1 - 1);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double2 a = t.T1[kc_wrap((long long)m1 * (q + 1), t.N1)];
      twa[q] = a.x;
      twb[q] = a.y;
    }
  }
  // H of both rows from one table: e the terms of even n1, o those of odd.
  auto eval = [&](const double* tb, double (&D)[2], double (&ox)[2], double (&oy)[2]) {
    const double2 z0 = *reinterpret_cast<const double2*>(tb);
    double e[3] = {z0.x, z0.y, tb[2]}, o[3];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double2 a = *reinterpret_cast<const double2*>(tb + 4 + 6 * q + 2 * i);
        if (q == 0)
          o[i] = fma(twa[q], a.x, twb[q] * a.y);
        else if (q % 2 == 1)
          e[i] = fma(twa[q], a.x, fma(twb[q], a.y, e[i]));
        else
          o[i] = fma(twa[q], a.x, fma(twb[q], a.y, o[i]));
      }
    }
    D[0] = e[0] + o[0];
    D[1] = e[0] - o[0];
    ox[0] = e[1] + o[1];
    ox[1] = e[1] - o[1];
    oy[0] = e[2] + o[2];
    oy[1] = e[2] - o[2];
  };
  // H of a step at its three points (real-space solver: [1] is twice H at t + dt/2).
  struct Hs {
    double D[3][2], x[3][2], y[3][2];
  };
  auto load = [&](const double* tb, Hs& h) {
    if constexpr (KM) {
      eval(tb, h.D[1], h.x[1], h.y[1]);
      eval(tb + TBL, h.D[2], h.x[2], h.y[2]);
    } else {
      eval(tb, h.D[0], h.x[0], h.y[0]);
      eval(tb + TBL, h.D[2], h.x[2], h.y[2]);
    }
  };
  auto step = [&](Hs& h) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if constexpr (KM) {
        h.D[0][j] = hD[j];
        h.x[0][j] = hx[j];
        h.y[0][j] = hy[j];
        hD[j] = h.D[2][j];
        hx[j] = h.x[2][j];
        hy[j] = h.y[2][j];
      } else {
        h.D[1][j] = h.D[0][j] + h.D[2][j];
        h.x[1][j] = h.x[0][j] + h.x[2][j];
        h.y[1][j] = h.y[0][j] + h.y[2][j];
      }
    }
    // RK4 (src/solver.cpp:157-163): X = rho + c k~, the middle stages' k~ twice k in the real-space solver;
    // kd = k00 / 2, k01 = (ty, -tx).
    const double c0 = 0.5 * dt, cm = KM ? 0.5 * dt : 0.25 * dt, ce = KM ? dt : 0.5 * dt;
    double d[2], xd[2], xx[2], xy[2], kd[2], tx[2], ty[2], sd[2], sx[2], sy[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      xd[j] = d[j] = r00[j] - r11[j];
      xx[j] = ux[j];
      xy[j] = uy[j];
    }
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      const int p = st == 0 ? 0 : (st == 3 ? 2 : 1);
      const double c = st == 0 ? c0 : (st == 1 ? cm : ce);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        kd[j] = h.x[p][j] * xy[j];
        tx[j] = xd[j] * h.x[p][j];
        ty[j] = xd[j] * h.y[p][j];
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        kd[j] = fma(h.y[p][j], xx[j], -kd[j]);
        tx[j] = fma(h.D[p][j], xx[j], -tx[j]);
        ty[j] = fma(h.D[p][j], xy[j], -ty[j]);
      }
      if (st < 3) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          xd[j] = fma(4.0 * c, kd[j], d[j]);
          xx[j] = fma(c, ty[j], ux[j]);
          xy[j] = fma(-c, tx[j], uy[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (st == 0) {
          sd[j] = kd[j];
          sx[j] = tx[j];
          sy[j] = ty[j];
        } else if (KM && st < 3) {
          sd[j] = fma(2.0, kd[j], sd[j]);
          sx[j] = fma(2.0, tx[j], sx[j]);
          sy[j] = fma(2.0, ty[j], sy[j]);
        } else {
          sd[j] += kd[j];
          sx[j] += tx[j];
          sy[j] += ty[j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      r00[j] = fma(2.0 * prefac, sd[j], r00[j]);
      r11[j] = fma(-2.0 * prefac, sd[j], r11[j]);
      ux[j] = fma(prefac, sy[j], ux[j]);
      uy[j] = fma(-prefac, sx[j], uy[j]);
    }
  };
  // Staged for the current: sums and differences of the pair (absent rows stay zero: their state is 0 and the
  // commutator keeps it there).
  auto stage = [&](int s, int b) {
    S.y[b][0][2 * s][lane] = r00[0] + r00[1];
    S.y[b][1][2 * s][lane] = r00[0] - r00[1];
    S.y[b][2][2 * s][lane] = r11[0] + r11[1];
    S.y[b][3][2 * s][lane] = r11[0] - r11[1];
    S.y[b][0][2 * s + 1][lane] = ux[0] + ux[1];
    S.y[b][1][2 * s + 1][lane] = ux[0] - ux[1];
    S.y[b][2][2 * s + 1][lane] = uy[0] + uy[1];
    S.y[b][3][2 * s + 1][lane] = uy[0] - uy[1];
  };
  auto last_sums = [&](int iv) {
    clear();
#pragma unroll
    for (int s = 0; s < kIv; ++s) sum_part(s, iv & 1);
    finish(iv);
  };
  asm volatile("cp.async.wait_all;" ::: "memory");
  sync();
  if (KM && steps) eval(S.cb, hD, hx, hy);

  for (int iv = 0; iv < nint; ++iv) {
    const int b = iv & 1, ns = min(kIv, step1 - step0 - iv * kIv);
    const double(*rec)[TT::REC] = S.rb[iv % 3];
    if (sums && iv + 1 < nint) fetch(iv + 1);
    if (SPLIT && sums) {
      last_sums(iv - 1);
    } else {
      if (!SPLIT) clear();
      // A whole interval unrolled.  The next step's H and the previous interval's sums come before this step's
      // stores (their loads could not pass them); neither depends on the state.
      Hs h[2];
      load(rec[0], h[0]);
      if (ns == kIv) {
#pragma unroll
        for (int s = 0; s < kIv; ++s) {
          if (s + 1 < kIv) load(rec[s + 1], h[(s + 1) & 1]);
          if (!SPLIT) {
            sum_part(s, b ^ 1);
            if (s + 1 == kIv) finish(iv - 1);
          }
          step(h[s & 1]);
          stage(s, b);
        }
      } else {
        if (!SPLIT) {
#pragma unroll
          for (int s = 0; s < kIv; ++s) sum_part(s, b ^ 1);
          finish(iv - 1);
        }
#pragma unroll 1
        for (int s = 0; s < ns; ++s) {
          if (s > 0) load(rec[s], h[0]);
          step(h[0]);
          stage(s, b);
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    sync();
  }
  if (sums) last_sums(nint - 1);
  auto put = [&](size_t k, int j) {
    A.rho[k * 4] = make_double2(r00[j], 0.0);
    A.rho[k * 4 + 1] = make_double2(ux[j], uy[j]);
    A.rho[k * 4 + 2] = make_double2(ux[j], -uy[j]);
    A.rho[k * 4 + 3] = make_double2(r11[j], 0.0);
  };
  if (on0) put(k0, 0);
  if (on1) put(k1, 1);
}

template <int Q, bool KM>
union KcolSmem {
  PropSmem<Q, KM> prop;
  TabSmem<Q, KM> tab;
};

template <int Q, bool KM, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 64 : 32, SPLIT ? 4 : 8) propagate_kcol_kernel(const __grid_constant__ KcolArgs A) {
  extern __shared__ __align__(16) unsigned char smraw[];
  KcolSmem<Q, KM>& S = *reinterpret_cast<KcolSmem<Q, KM>*>(smraw);
  if ((int)blockIdx.x >= A.nprop) {
    const int idx = blockIdx.x - A.nprop;
    if (SPLIT && threadIdx.x >= 32) return;
    column_tables<Q, KM>(A.t, A.gt, A.next0, A.next1, idx % A.t.N2, idx / A.t.N2 * kTabPts, A.chunk, A.next, S.tab);
    return;
  }
  // Virtual CTA v owns tiles v, v + vctas, ... and its own row of current partials.
  const int pairs = min(A.t.row1 - A.t.row0, A.t.N1 / 2), ntiles = A.t.N2 * ((pairs + A.R - 1) / A.R);
  for (int v = blockIdx.x; v < A.vctas; v += A.nprop)
    for (int tile = v; tile < ntiles; tile += A.vctas) propagate_tile<Q, KM, SPLIT>(A, v, tile, S.prop);
}

using KcolKernel = void (*)(const KcolArgs);
struct Form {
  KcolKernel kern[2];     // one warp per tile, two
  size_t smem, rec, col;  // bytes; doubles per step and column of the tables
};
template <int Q, bool KM>
constexpr Form form_t() {
  return {{propagate_kcol_kernel<Q, KM, false>, propagate_kcol_kernel<Q, KM, true>}, sizeof(KcolSmem<Q, KM>), Tables<Q, KM>::REC, Tables<Q, KM>::COL};
}
Form form_of(const SolveTables& t) {
  if (std::max(t.b1n, t.b2n) > 5) return t.kmode ? form_t<3, true>() : form_t<3, false>();
  return t.kmode ? form_t<2, true>() : form_t<2, false>();
}
constexpr int kPairVariant = 2;  // LaunchShape::variant of this kernel (0, 1: sbe_kcol_any.cu)

}  // namespace

bool plan_kcol(const SolveTables& t, int sm_count, LaunchShape* out, size_t smem_max, int parts_hint) {
  const char* full = std::getenv("HHG_KCOL_FULLBOX");
  const bool symmetric = t.b1n % 2 == 1 && t.b1lo == -(t.b1n - 1) / 2 && t.b2n % 2 == 1 && t.b2lo == -(t.b2n - 1) / 2;
  if (t.nw != 2 || !t.hermitian || !symmetric || t.nj > kNj || t.b1n > 7 || t.b2n > 7 || (full && full[0] == '1'))
    return plan_kcol_any(t, sm_count, out, smem_max, parts_hint);
  // Tiles of equal parts of a column of at most 32 pairs.
  const int pairs = std::min(t.row1 - t.row0, t.N1 / 2), least = (pairs + 31) / 32;
  int parts = std::max(least, parts_hint);
  if (const char* e = std::getenv("HHG_KCOL_PARTS")) parts = std::max(least, std::atoi(e));  // tuning override
  const int R = (pairs + parts - 1) / parts;
  const long ntiles = (long)t.N2 * ((pairs + R - 1) / R);
  const Form f = form_of(t);
  // Two warps a tile up to 1.5 tiles an SM: 1024 steps of a 20 x 20 grid (20 tiles) 0.27 ms against 0.38 with one,
  // 100 x 100 (200 tiles) 0.31 against 0.39; beyond, the second warps' registers and barriers cost more than they
  // hide: 120 x 120 (240 tiles) 0.45 against 0.40, 200 x 200 (800 tiles, 4096 steps) 2.90 against 2.60.
  const int warps = 2 * ntiles <= 3 * sm_count ? 2 : 1;
  const KcolKernel kern = f.kern[warps - 1];
  allow_shared_memory(kern, f.smem);
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * warps, f.smem);
  if (occ < 1) return plan_kcol_any(t, sm_count, out, smem_max, parts_hint);
  const long slots = (long)occ * sm_count;
  out->kernel = 3;
  out->kmode = t.kmode;
  out->k_per_cta = 2 * R;
  out->group = 1;
  out->threads = 32 * warps;
  out->ntiles = (int)ntiles;
  out->ctas = (int)(ntiles < slots ? ntiles : slots);
  out->vctas = out->ctas;
  out->box_sm = out->win_sm = 0;
  out->ept = 1;
  out->variant = kPairVariant;
  out->smem = f.smem;
  out->pre_chunk = std::min(kKcolChunk, t.nt);
  out->pre_bytes = 2 * 8 * (size_t)t.N2 * (out->pre_chunk * f.rec + f.col);
  return true;
}

int launch_kcol(const SolveTables& t, const GroupTables& gt, const LaunchShape& s, double2* rho, double2* Jpart,
                cudaStream_t stream) {
  if (s.variant != kPairVariant) {
    launch_kcol_any(t, gt, s, rho, Jpart, stream);
    return 1;
  }
  if (!gt.pre || s.pre_chunk <= 0)
    throw std::runtime_error("column-tile launch: needs its table scratch (GroupTables::pre)");
  const Form f = form_of(t);
  const KcolKernel kern = f.kern[s.threads / 32 - 1];
  allow_shared_memory(kern, s.smem);
  double* tables[2] = {static_cast<double*>(gt.pre), static_cast<double*>(gt.pre) + (size_t)t.N2 * (s.pre_chunk * f.rec + f.col)};
  KcolArgs a{};
  a.t = t;
  a.gt = gt;
  a.chunk = s.pre_chunk;
  a.R = s.k_per_cta / 2;
  a.vctas = s.vctas;
  a.rho = rho;
  a.Jpart = Jpart;
  int launches = 0;
  // The first launch forms the first chunk's tables only; each later one propagates a chunk and forms the next's.
  for (int c0 = t.step0 - s.pre_chunk; c0 < t.step1; c0 += s.pre_chunk) {
    a.next0 = std::min(c0 + s.pre_chunk, t.step1);
    a.next1 = std::min(a.next0 + s.pre_chunk, t.step1);
    a.next = tables[launches & 1];
    a.cur = tables[(launches + 1) & 1];
    a.nprop = launches == 0 ? 0 : s.ctas;
    a.t.step0 = c0;
    a.t.step1 = a.next0;
    const int pts = (t.kmode ? 2 : 1) * (a.next1 - a.next0), groups = (pts + kTabPts - 1) / kTabPts;
    kern<<<a.nprop + groups * t.N2, s.threads, s.smem, stream>>>(a);
    ++launches;
  }
  return launches;
}

}  // namespace hhg
