// FP64 tensor-core form of the plain propagation for 3..12 orbitals.
//
// Same propagation as group_vctas (sbe_group.cu) in FP64 (k-space-resident RK4 of the reference's
// src/solver.cpp:86-181, 1428-1726, and the windowed current of src/observable.cpp:16-30; the k-space
// solver of src/solver_kspace.cpp:167-270 as KM), for Hermitian placements with a cell box symmetric
// about zero and at most 7 cells high.  All products run on the FP64 tensor cores (mma.m8n8k4.f64: IEEE
// double products and sums).  FP64 products and the FP64 units share one pipe per SM sub-partition (16
// cycles per m8n8k4, 2 per FP64 warp instruction), and that pipe bounds the kernel, so every form below
// is the one that asks least of it.
//
// Layout.  A warp holds KPW k-points.  rho and every H and k are Hermitian, and lane (g = lane / 4,
// c = lane % 4; h = g / 2, p = g % 2) holds of each matrix M
//    T[e] = M[g][2c + e]           (complex, e = 0, 1)   the 8 x 8 block of orbitals 0..7
// and, with 9..12 orbitals (BIG),
//    U    = M[g][8 + c]            (complex)
//    L[e] = part p of M[2c + e][8 + h]   (real: p = 0 real part, p = 1 imaginary)
//    V    = part p of M[8 + c][8 + h]    (real)
// L is U transposed as an 8 x 8 block of reals, so a state is T, U, V: 7 doubles a lane.  The real and
// imaginary parts of orbitals 8..11 sit side by side in the 8 rows or columns of one product, which
// therefore wastes nothing on 12 orbitals: a commutator is 24 m8n8k4 (a 16 x 16 frame: 36).
//
//  * [H, X], block (0..7, 0..7): P = H X with three real products per complex one (Gauss), k = -i (P - P^+),
//    P^+ by register transposes;
//  * block (0..7, 8..11): H X - X H in full, the second operand's parts stacked over its columns (L, V);
//  * block (8..11, 8..11): the parts stacked over rows and columns, two shuffles for P - P^+.
//
// H(k) at the step's three field samples.  M(k) = sum_n1 p(n1) G(n1) over the box rows with
// G(-n1) = G(n1)^+ and p(-n1) = conj p(n1) is a real product: with p = a + ib,
//    Re M_ij = a0 G0.x + sum_{n1 > 0} (a S.x - b D.y),  Im M_ij = a0 G0.y + sum (a S.y + b D.x),
//    S = G_ij + conj G_ji,  D = G_ij - conj G_ji,
// so the CTA's k-points (rows) times the real and imaginary parts of the elements i <= j (columns) take
// 2 k-steps [a0 0 a1 b1 | a2 b2 a3 b3] per 8 x 8 tile.  dfrag_sums_kernel forms the S and D columns of a
// chunk of 64 steps in operand order, once per k-grid column; the field is applied to the accumulators.
//
// Current: J_a = sum_q sum_n coef(a, q, n) Z(q, n) with Z(q, n) = sum_k wp(k, q) x_n(k) over the real and
// imaginary parts x_n of the elements i <= j of rho(k): a product [4 window rows x 2 parts] x [k-points] x
// [elements x 2 parts] per CTA and step, contracted with the column's window coefficients (written by
// dfrag_sums_kernel) after the k-sum.
//
// A step has two phases between CTA barriers: the RK4 stages (each warp its own k-points), and the
// current of the step (NCW warps) beside the H of the next one (the others).
//
// Measured on B200 (1965 MHz): 11 orbitals, 150 x 150, one field axis, 4096 steps 262 ms (a 16 x 16 frame with
// one k-point per warp at 208 registers, 8 warps per SM: 525 ms); 6 orbitals, 100 x 100, two axes, 4096 steps
// 52.2 ms (element-group kernel 162 ms); 12 orbitals, 64 x 64, two axes, k-space solver, 1024 steps 17.1 ms
// (element groups 72.6); 5 orbitals, 46 x 38, 1024 steps 3.7 ms (element groups 9.5).  The shared FP64/tensor
// pipe is 81-83 % busy.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>

#include "dmma.cuh"
#include "sbe_device.h"
#include "smem_limit.h"
#include "warp_reduce.cuh"

namespace hhg {
namespace {

constexpr int kDfWarps = 8, kDfThreads = kDfWarps * 32;
constexpr int kDfKS = 2;         // k-steps of the outer sums: box half-heights up to 3
constexpr int kDfChunk = 64;     // steps per sums + propagation launch pair
constexpr int kDfRing = 16;      // steps per flush of the current partials
constexpr int kDfNj = 2;         // current axes
constexpr int kDfMaxBox2 = 64;   // widest cell box along the second axis
constexpr int kDfSumPts = 4;     // points per block of the sums kernel
constexpr int kDfSumThreads = 192;

__device__ __forceinline__ double2 df_mul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 df_fmac(double2 a, double2 b, double2 c) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
  return c;
}
__device__ __forceinline__ int df_wrap(long long x, int n) {
  const int r = (int)(x % n);
  return r < 0 ? r + n : r;
}
__device__ __forceinline__ double df_flip(double x, unsigned sign) {
  return __hiloint2double(__double2hiint(x) ^ (int)sign, __double2loint(x));
}
template <int BYTES>
__device__ __forceinline__ void df_cp_async(void* dst_smem, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void df_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Element (i <= j) of a Hermitian matrix: packed upper triangle by columns, the same for any orbital count.
__host__ __device__ constexpr int df_elem(int i, int j) { return j * (j + 1) / 2 + i; }

// Window coefficients read through L1 instead of staged: the k-space solver's are the same for all steps, and with
// 9..12 orbitals and two axes staging them leaves one CTA on an SM at 12 orbitals (64 x 64, 1024 steps: 20.5 ms
// staged, 17.0 not; 11 orbitals, where both fit twice, 8.0 and 8.1 for 512 steps).
__host__ __device__ constexpr bool df_coef_global(bool big, int nax, bool km) { return km && big && nax >= 2; }

// Shapes shared by the kernels and the planner (nt: 8-column tiles of the elements' parts).
struct DfLayout {
  int nt, hks, rhos;   // double2 per k-point and sample of H; doubles per k-point of the staged state
  size_t gpt, wpt;     // doubles of one point's sums and window coefficients per column
  size_t HK, GB, CW, RHO, TW1, WTW1, PQ, PW, ES, SJ, bytes;
  __host__ __device__ DfLayout(int nw, int nax, int nj, int kpc, bool km, int ncw) {
    nt = (nw * (nw + 1) + 7) / 8;
    hks = 4 * nt + 4;  // one zero slot past the elements; 4 mod 8 keeps the tile stores conflict-free
    if (hks % 8 != 4) hks += 4;
    rhos = 8 * nt + 4;  // 4 or 12 mod 16: conflict-free operand loads
    gpt = (size_t)(1 + nax) * nt * kDfKS * 32;
    wpt = (size_t)nj * nt * 64;
    size_t b = 0;
    HK = b;
    b += (size_t)3 * kpc * hks * 16;
    GB = b;
    b += (km ? 2 : 1) * gpt * 8;
    CW = b;
    if (!df_coef_global(nw > 8, nax, km)) b += wpt * 8;
    RHO = b;
    b += (size_t)kpc * rhos * 8;
    TW1 = b;
    b += (size_t)kpc * 4 * 16;
    WTW1 = b;
    b += (size_t)kpc * 4 * 16;
    PQ = b;
    b += 2 * 4 * 16;
    PW = b;
    b += 4 * 16;
    ES = b;
    b += 10 * 8;
    SJ = b;
    b += (size_t)kDfRing * ncw * 6 * 8;
    bytes = (b + 15) / 16 * 16;
  }
};

struct DfData {
  const double2 *Xbox, *Xwin, *P, *T1, *T2;
  const double* GB;  // [point][N2][1 + nax][nt][kDfKS][32]
  const double* CW;  // [point][N2][nj][nt][16][4] (k-space solver: [N2]...)
};

// The sums of every column for the chunk's points: block = (kDfSumPts points, column).  A thread forms, for one
// matrix, element pair (i, j), (j, i) and box row n1, the column sums G(n1) = sum_n2 p2(n2) X(n1, n2) at the
// block's points.  It is bound by the latency of the table loads, so a thread keeps few accumulators and many
// warps fit: with two rows and eight points per thread (168 registers) the chunk took 1.4 times as long.
__global__ void __launch_bounds__(kDfSumThreads, 4) dfrag_sums_kernel(SolveTables t, DfData d, int nt, double* GB,
                                                                      double* CW, int npts) {
  constexpr int P = kDfSumPts;
  __shared__ double2 q2[P][kDfMaxBox2];
  __shared__ double2 w2[P][4];
  const int m2 = blockIdx.x, sl0 = blockIdx.y * P, ns = min(P, npts - sl0);
  const int npw = 2 * t.np + 1, W1n = t.b1n, W2n = t.b2n, nw = t.nw, nw2 = t.nw2, half = (W1n - 1) / 2;
  const int nmat = 1 + t.nax, ne = nw * (nw + 1) / 2, ne4 = 4 * nt;
  for (int idx = threadIdx.x; idx < P * (W2n + 4); idx += blockDim.x) {
    const int j = idx / (W2n + 4), q = idx % (W2n + 4);
    const int s = (t.kmode ? 2 * t.step0 : t.step0) + sl0 + min(j, ns - 1);
    const double2* P2 = d.P + (size_t)s * 2 * npw + t.np + npw;
    if (q < W2n) {
      q2[j][q] = df_mul(d.T2[df_wrap((long long)m2 * (t.b2lo + q), t.N2)], P2[t.b2lo + q]);
    } else {
      const int qw = q - W2n;
      const double2 tw = d.T2[df_wrap((long long)m2 * (qw - 2), t.N2)];
      w2[j][qw] = t.kmode ? tw : df_mul(tw, P2[qw - 2]);
    }
  }
  __syncthreads();
  const double2 zero = make_double2(0.0, 0.0);
  const size_t gpt = (size_t)nmat * nt * kDfKS * 32, wpt = (size_t)t.nj * nt * 64;
  // Column j of packed element e (padding past ne: an empty element).
  auto column = [&](int e) {
    int j = 0;
    while (df_elem(0, j + 1) <= e) ++j;
    return j;
  };
  for (int idx = threadIdx.x; idx < 4 * nmat * ne4; idx += blockDim.x) {
    // (neighbouring threads take the two rows n1 = q of a k-step: their 16-byte stores share a sector)
    const int qs = idx & 1, e = (idx >> 1) % ne4, mk = (idx >> 1) / ne4, ks = mk & 1, mat = mk >> 1, q = 2 * ks + qs;
    const int j = column(e), i = e - df_elem(0, j);
    const bool on = e < ne && q <= half;
    const double2* X = d.Xbox + (size_t)(mat * W1n + half + (on ? q : 0)) * W2n * nw2;
    const int o0 = on ? i * nw + j : 0, o1 = on ? j * nw + i : 0;
    double2 a[P], b[P];  // G(q) of (i, j) and of (j, i)
#pragma unroll
    for (int s = 0; s < P; ++s) a[s] = b[s] = zero;
    if (on) {
      double2 x = X[o0], y = X[o1];
#pragma unroll 1
      for (int n = 0; n < W2n; ++n) {
        // (the next cell's table values are on their way while this one's are used)
        const int n1 = min(n + 1, W2n - 1) * nw2;
        const double2 xn = X[n1 + o0], yn = X[n1 + o1];
#pragma unroll
        for (int s = 0; s < P; ++s) {
          const double2 pf = q2[s][n];
          a[s] = df_fmac(pf, x, a[s]);
          b[s] = df_fmac(pf, y, b[s]);
        }
        x = xn;
        y = yn;
      }
    }
    double* dst = GB + ((size_t)sl0 * t.N2 + m2) * gpt + (((size_t)mat * nt + e / 4) * kDfKS + ks) * 32 + 8 * (e % 4) + 2 * qs;
#pragma unroll
    for (int s = 0; s < P; ++s)
      if (s < ns) {
        double2* o = reinterpret_cast<double2*>(dst + (size_t)s * t.N2 * gpt);
        if (q == 0) {
          o[0] = make_double2(a[s].x, 0.0);
          o[2] = make_double2(i == j ? 0.0 : a[s].y, 0.0);
        } else {
          o[0] = make_double2(a[s].x + b[s].x, -(a[s].y + b[s].y));
          o[2] = make_double2(a[s].y - b[s].y, a[s].x - b[s].x);
        }
      }
  }
  // Window coefficients of the parts (x, y) of element i <= j: x multiplies GW_ij + GW_ji, y multiplies
  // -i (GW_ij - GW_ji).
  const int nwp = t.kmode ? (sl0 == 0 ? 1 : 0) : ns;  // points whose window this block writes
  for (int idx = threadIdx.x; nwp > 0 && idx < t.nj * 4 * ne4; idx += blockDim.x) {
    const int e = idx % ne4, aq = idx / ne4;
    const int j = column(e), i = e - df_elem(0, j);
    // (the sums are linear in the tables: x and y of the window first)
    double2 x[4], y[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const double2 u = e < ne ? d.Xwin[(size_t)(aq * 4 + n) * nw2 + i * nw + j] : zero;
      const double2 v = e < ne && i != j ? d.Xwin[(size_t)(aq * 4 + n) * nw2 + j * nw + i] : zero;
      x[n] = make_double2(u.x + v.x, u.y + v.y);
      y[n] = i == j ? zero : make_double2(u.y - v.y, v.x - u.x);
    }
#pragma unroll 2
    for (int s = 0; s < nwp; ++s) {
      double2 a = zero, b = zero;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        a = df_fmac(w2[s][n], x[n], a);
        b = df_fmac(w2[s][n], y[n], b);
      }
      const size_t blk = t.kmode ? (size_t)m2 : (size_t)(sl0 + s) * t.N2 + m2;
      double2* dst = reinterpret_cast<double2*>(CW + blk * wpt + (((size_t)(aq / 4) * nt + e / 4) * 16 + (aq % 4) * 4 + e % 4) * 4);
      dst[0] = a;
      dst[1] = b;
    }
  }
}

__host__ __device__ constexpr int df_current_warps(bool big, bool km) { return big || km ? 4 : 5; }

// BIG: 9..12 orbitals (one k-point per warp, 8 per CTA); otherwise 3..8 (two per warp, 16 per CTA).
template <bool BIG, int NAX, bool KM>
struct DfShape {
  static constexpr int KPW = BIG ? 1 : 2, KPC = kDfWarps * KPW, MT = KPC / 8;
  // Warps that form the current; the others form the next step's H.  A tile of the current (KPC / 4 products,
  // four FP64 operations per axis and part) takes about twice a tile of H.  11 orbitals, 1024 steps of 150 x 150:
  // 69.2 ms with 3, 66.0 with 4; 6 orbitals, 100 x 100: 54.1 with 3, 52.9 with 5, 54.8 with 6; 12 orbitals, k-space
  // solver: 22.2 with 2, 20.8 with 4.
  static constexpr int NCW = df_current_warps(BIG, KM);
};

template <bool BIG, int NAX, bool KM>
__global__ void __launch_bounds__(kDfThreads, 2)
    propagate_dfrag_kernel(SolveTables t, DfData d, int vctas, double2* rho, double2* Jpart) {
  using SH = DfShape<BIG, NAX, KM>;
  constexpr int KPW = SH::KPW, KPC = SH::KPC, MT = SH::MT, NCW = SH::NCW, NOW = kDfWarps - NCW, NMAT = 1 + NAX;
  constexpr int NB = BIG ? 3 : 2;  // k-steps of the commutator: columns 2c, 2c + 1 (and 8 + c)
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nw = t.nw, nw2 = t.nw2, nj = t.nj;
  const DfLayout L(nw, NAX, nj, KPC, KM, NCW);
  const int nt = L.nt, hks = L.hks, rhos = L.rhos;
  double2* HK = reinterpret_cast<double2*>(smraw + L.HK);
  double* GB = reinterpret_cast<double*>(smraw + L.GB);
  double* CW = reinterpret_cast<double*>(smraw + L.CW);
  double* RHO = reinterpret_cast<double*>(smraw + L.RHO);
  double2* TW1 = reinterpret_cast<double2*>(smraw + L.TW1);
  double2* WTW1 = reinterpret_cast<double2*>(smraw + L.WTW1);
  double2* PQ = reinterpret_cast<double2*>(smraw + L.PQ);
  double2* PW = reinterpret_cast<double2*>(smraw + L.PW);
  double* ES = reinterpret_cast<double*>(smraw + L.ES);
  double* SJ = reinterpret_cast<double*>(smraw + L.SJ);

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, c4 = lane & 3, h = g >> 1, p = g & 1;
  const int rows = t.row1 - t.row0, bpc = (rows + KPC - 1) / KPC, ntiles = t.N2 * bpc;
  const int step0 = t.step0, step1 = t.step1, npw = 2 * t.np + 1, half = (t.b1n - 1) / 2;
  const double dt = t.dt, prefac = 0.1666666666666 * dt;
  const double2 zero = make_double2(0.0, 0.0);
  const unsigned psign = (unsigned)p << 31;

  // This lane's elements in the packed triangle (the zero slot where an orbital is missing) and the signs
  // of their imaginary parts.
  const int ze = 4 * nt;
  int eT[2], eU = ze, eL[2] = {ze, ze}, eV = ze;
  unsigned sT[2], sV = 0u;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int col = 2 * c4 + e;
    eT[e] = (g < nw && col < nw) ? (g <= col ? df_elem(g, col) : df_elem(col, g)) : ze;
    sT[e] = g > col ? 0x80000000u : 0u;
  }
  if constexpr (BIG) {
    if (8 + c4 < nw) eU = df_elem(g, 8 + c4);
    if (8 + h < nw) {
#pragma unroll
      for (int e = 0; e < 2; ++e) eL[e] = df_elem(2 * c4 + e, 8 + h);
      if (8 + c4 < nw) {
        eV = c4 <= h ? df_elem(8 + c4, 8 + h) : df_elem(8 + h, 8 + c4);
        sV = c4 > h ? psign : 0u;
      }
    }
  }
  const int vsrc = (2 * c4 + p) * 4 + h;  // the lane of the transposed element of block (8..11, 8..11)
  // H sample of evaluation point offset f (0, 1, 2: t, t + dt/2, t + dt) of step ti.
  auto slot_of = [&](int ti, int f) { return KM ? (f == 1 ? 2 : (ti + (f >> 1)) & 1) : f; };

  for (int idx = tid; idx < 3 * KPC * hks; idx += kDfThreads) HK[idx] = zero;
  for (int idx = tid; idx < KPC * rhos; idx += kDfThreads) RHO[idx] = 0.0;

  for (int v = blockIdx.x; v < vctas; v += gridDim.x)
    for (int tile = v; tile < ntiles; tile += vctas) {
      const int m2 = tile / bpc, m10 = t.row0 + (tile % bpc) * KPC;
      const int nown = min(KPC, t.row1 - m10);

      // Sums of point pt into GB slot pb, with its row factors.
      auto fetch_point = [&](int pt, int pb) {
        const double* src = d.GB + ((size_t)(pt - (KM ? 2 * step0 : step0)) * t.N2 + m2) * L.gpt;
        double* dst = GB + pb * L.gpt;
        for (int idx = tid; idx < (int)L.gpt / 2; idx += kDfThreads) df_cp_async<16>(dst + 2 * idx, src + 2 * idx);
        if (tid <= half) df_cp_async<16>(PQ + 4 * pb + tid, d.P + (size_t)pt * 2 * npw + t.np + tid);
      };
      auto fetch_window = [&](int ti) {
        const double* src = d.CW + (KM ? (size_t)m2 : (size_t)(ti - step0) * t.N2 + m2) * L.wpt;
        for (int idx = tid; idx < (int)L.wpt / 2; idx += kDfThreads) df_cp_async<16>(CW + 2 * idx, src + 2 * idx);
        if (!KM && tid < 4) df_cp_async<16>(PW + tid, d.P + (size_t)ti * 2 * npw + t.np + tid - 2);
      };
      auto fetch_field = [&](int ti) {
        if (tid < 9) df_cp_async<8>(ES + tid, t.es + (size_t)ti * 9 + tid);
      };
      // H of step ti from the sums in GB, by warps wo = 0 .. nwo - 1.  RS: one point, three field samples;
      // KM: points t + dt/2 and t + dt (first: the chunk's point t from slot 0).
      auto outer = [&](int ti, bool first, int wo, int nwo) {
        double ea[3][NAX];
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
          for (int a = 0; a < NAX; ++a) ea[f][a] = ES[f * 3 + t.ax_id[a]];
        constexpr int NPT = KM ? 2 : 1;
#pragma unroll
        for (int pb = 0; pb < NPT; ++pb) {
          if (KM && first && pb == 1) break;
          double pa[MT][2];  // A[g][c] of the k-steps: part c % 2 of p(n1 = c / 2), p(n1 = 2 + c / 2) of k-point 8 m + g
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              const int q = 2 * ks + (c4 >> 1);
              const double2 tw = TW1[(8 * m + g) * 4 + q], pq = PQ[4 * pb + q];
              pa[m][ks] = q > half ? 0.0 : (c4 & 1) ? fma(tw.x, pq.y, tw.y * pq.x) : fma(tw.x, pq.x, -tw.y * pq.y);
            }
#pragma unroll 2
          for (int n = wo; n < nt; n += nwo) {
            double acc[NMAT][MT][2];
#pragma unroll
            for (int mat = 0; mat < NMAT; ++mat)
#pragma unroll
              for (int m = 0; m < MT; ++m) acc[mat][m][0] = acc[mat][m][1] = 0.0;
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
              for (int mat = 0; mat < NMAT; ++mat) {
                const double b = GB[pb * L.gpt + (((size_t)mat * nt + n) * kDfKS + ks) * 32 + lane];
#pragma unroll
                for (int m = 0; m < MT; ++m) dmma(acc[mat][m], pa[m][ks], b);
              }
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                if (KM && f != (first ? 0 : 1 + pb)) continue;
                double2 hv = make_double2(acc[0][m][0], acc[0][m][1]);
#pragma unroll
                for (int a = 0; a < NAX; ++a) {
                  hv.x = fma(ea[f][a], acc[1 + a][m][0], hv.x);
                  hv.y = fma(ea[f][a], acc[1 + a][m][1], hv.y);
                }
                HK[((size_t)slot_of(ti, f) * KPC + 8 * m + g) * hks + 4 * n + c4] = hv;
              }
          }
        }
      };
      // Current partials of step ti, by warps wc = 0 .. NCW - 1.
      auto current = [&](int ti, int wc) {
        double wa[KPC / 4];  // A[g][c]: part p of wp(k-point 4 ks + c, window row h)
        {
          const double2 pw = KM ? make_double2(1.0, 0.0) : PW[h];
#pragma unroll
          for (int ks = 0; ks < KPC / 4; ++ks) {
            const double2 tw = WTW1[(4 * ks + c4) * 4 + h];
            wa[ks] = p ? fma(tw.x, pw.y, tw.y * pw.x) : fma(tw.x, pw.x, -tw.y * pw.y);
          }
        }
        double u[3] = {0.0, 0.0, 0.0}, s[3] = {0.0, 0.0, 0.0};
        const double* rb = RHO + c4 * rhos + g;
        constexpr bool CG = df_coef_global(BIG, NAX, KM);
        const double* cw = (CG ? d.CW + (size_t)m2 * L.wpt : CW) + (h * 4 + c4) * 4;
#pragma unroll 2
        for (int n = wc; n < nt; n += NCW) {
          double z[2] = {0.0, 0.0};
#pragma unroll
          for (int ks = 0; ks < KPC / 4; ++ks) dmma(z, wa[ks], rb[4 * ks * rhos + 8 * n]);
#pragma unroll
          for (int a = 0; a < kDfNj; ++a)
            if (a < nj) {
              const double2* cf = reinterpret_cast<const double2*>(cw + (a * nt + n) * 64);
              const double2 cx = CG ? __ldg(cf) : cf[0], cy = CG ? __ldg(cf + 1) : cf[1];
              u[a] = fma(cx.x, z[0], fma(cy.x, z[1], u[a]));
              s[a] = fma(cx.y, z[0], fma(cy.y, z[1], s[a]));
            }
        }
        double re[3], im[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          re[a] = p ? -s[a] : u[a];
          im[a] = p ? u[a] : s[a];
        }
        warp_store_current(re, im, nj, lane, SJ + ((ti % kDfRing) * NCW + wc) * 6);
      };
      // The partials of the ring's steps up to ti_end, into this virtual CTA's row.
      auto flush = [&](int ti_end) {
        const int ti0 = max(ti_end - ti_end % kDfRing, step0), nsteps = ti_end - ti0 + 1;
        for (int idx = tid; idx < nsteps * nj; idx += kDfThreads) {
          const int ti = ti0 + idx / nj, a = idx % nj;
          double re = 0.0, im = 0.0;
#pragma unroll
          for (int ww = 0; ww < NCW; ++ww) {
            re += SJ[((ti % kDfRing) * NCW + ww) * 6 + 2 * a];
            im += SJ[((ti % kDfRing) * NCW + ww) * 6 + 2 * a + 1];
          }
          const int ja = a == 0 ? t.j_id[0] : (a == 1 ? t.j_id[1] : t.j_id[2]);
          double2* dst = Jpart + ((size_t)v * t.nt + ti) * 3 + ja;
          const double2 old = *dst;
          *dst = make_double2(old.x + re, old.y + im);
        }
      };

      __syncthreads();  // the previous tile's readers of the tables are done
      for (int idx = tid; idx < KPC * 4; idx += kDfThreads) {
        const int m1 = min(m10 + idx / 4, t.row1 - 1), q = idx % 4;
        TW1[idx] = d.T1[df_wrap((long long)m1 * q, t.N1)];
        WTW1[idx] = d.T1[df_wrap((long long)m1 * (q - 2), t.N1)];
      }
      if (tid < 8) PQ[tid] = zero;
      __syncthreads();
      fetch_point(KM ? 2 * step0 : step0, 0);
      fetch_field(step0);
      if (KM && !df_coef_global(BIG, NAX, KM)) fetch_window(step0);
      // This warp's states.
      double2 rT[KPW][2], rU[KPW];
      double rV[KPW];
      bool kval[KPW];
#pragma unroll
      for (int kk = 0; kk < KPW; ++kk) {
        const int kp = w * KPW + kk;
        kval[kk] = kp < nown;
        const double2* src = rho + ((size_t)(m10 + (kval[kk] ? kp : 0)) * t.N2 + m2) * nw2;
#pragma unroll
        for (int e = 0; e < 2; ++e)
          rT[kk][e] = kval[kk] && eT[e] != ze ? src[g * nw + 2 * c4 + e] : zero;
        if constexpr (BIG) {
          rU[kk] = kval[kk] && eU != ze ? src[g * nw + 8 + c4] : zero;
          const double2 vv = kval[kk] && eV != ze ? src[(8 + c4) * nw + 8 + h] : zero;
          rV[kk] = p ? vv.y : vv.x;
        }
        if (!kval[kk])
          for (int idx = lane; idx < rhos; idx += 32) RHO[(size_t)kp * rhos + idx] = 0.0;
      }
      df_cp_wait();
      __syncthreads();
      outer(step0, KM, w, kDfWarps);
      __syncthreads();
      if constexpr (KM) {
        fetch_point(2 * step0 + 1, 0);
        fetch_point(2 * step0 + 2, 1);
        df_cp_wait();
        __syncthreads();
        outer(step0, false, w, kDfWarps);
        __syncthreads();
      }

      for (int ti = step0; ti < step1; ++ti) {
        if (ti > step0 && ti % kDfRing == 0) flush(ti - 1);
        // The next step's sums and field and this step's window coefficients: the buffers' last readers
        // finished before the barrier.
        if constexpr (!KM) fetch_window(ti);
        if (ti + 1 < step1) {
          if constexpr (KM) {
            fetch_point(2 * ti + 3, 0);
            fetch_point(2 * ti + 4, 1);
          } else {
            fetch_point(ti + 1, 0);
          }
          fetch_field(ti + 1);
        }

        // RK4 stages (src/solver.cpp:157-180), fields at t, t + dt/2, t + dt/2, t + dt.
        if (kval[0]) {
          double2 xT[KPW][2], xU[KPW], sT_[KPW][2], sU[KPW], hT[KPW][2], hU[KPW];
          double xV[KPW], sV_[KPW], hL[KPW][2], hV[KPW];  // hL, hV: negated
#pragma unroll
          for (int kk = 0; kk < KPW; ++kk) {
            xT[kk][0] = rT[kk][0];
            xT[kk][1] = rT[kk][1];
            sT_[kk][0] = sT_[kk][1] = zero;
            if constexpr (BIG) {
              xU[kk] = rU[kk];
              xV[kk] = rV[kk];
              sU[kk] = zero;
              sV_[kk] = 0.0;
            }
          }
#pragma unroll 1
          for (int st = 0; st < 4; ++st) {
            const int f = st == 0 ? 0 : (st == 3 ? 2 : 1);
            const double wgt = (st == 0 || st == 3) ? 1.0 : 2.0;
            const double cn = (st == 2 ? 1.0 : 0.5) * dt;
            if (st != 2) {  // (the third stage keeps the second's H)
#pragma unroll
              for (int kk = 0; kk < KPW; ++kk) {
                const double2* Hk = HK + ((size_t)slot_of(ti, f) * KPC + w * KPW + kk) * hks;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  hT[kk][e] = Hk[eT[e]];
                  hT[kk][e].y = df_flip(hT[kk][e].y, sT[e]);
                }
                if constexpr (BIG) {
                  hU[kk] = Hk[eU];
                  const double* Hd = reinterpret_cast<const double*>(Hk) + p;
#pragma unroll
                  for (int e = 0; e < 2; ++e) hL[kk][e] = -Hd[2 * eL[e]];
                  hV[kk] = df_flip(Hd[2 * eV], sV ^ 0x80000000u);
                }
              }
            }
#pragma unroll
            for (int kk = 0; kk < KPW; ++kk) {
              // Block (0..7, 0..7): A[g][k] = H[g][k], B[k][g] = conj(X[g][k]).
              double2 ha[NB], xa[NB];
              ha[0] = hT[kk][0];
              ha[1] = hT[kk][1];
              xa[0] = xT[kk][0];
              xa[1] = xT[kk][1];
              if constexpr (BIG) {
                ha[2] = hU[kk];
                xa[2] = xU[kk];
              }
              double t1[2] = {0.0, 0.0}, t2[2] = {0.0, 0.0}, t3[2] = {0.0, 0.0};
#pragma unroll
              for (int k = 0; k < NB; ++k) {
                dmma(t1, ha[k].x, xa[k].x);
                dmma(t2, ha[k].y, xa[k].y);
                dmma(t3, ha[k].x + ha[k].y, xa[k].x - xa[k].y);
              }
              double2 kU = zero;
              double kV = 0.0;
              if constexpr (BIG) {
                double xL[3] = {xU[kk].x, xU[kk].y, xV[kk]};
                transpose8(xL[0], xL[1]);
                const double hN[3] = {hL[kk][0], hL[kk][1], hV[kk]};
                // Block (0..7, 8..11): H X - X H, columns (8 + c, part).
                double b1[2] = {0.0, 0.0}, b2[2] = {0.0, 0.0}, dd[2] = {0.0, 0.0};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                  dmma(b1, xa[k].x, hN[k]);
                  dmma(b2, xa[k].y, hN[k]);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                  dmma(dd, hN[k], xL[k]);
                  dmma(b1, ha[k].x, xL[k]);
                  dmma(b2, ha[k].y, xL[k]);
                }
                kU = make_double2(b1[1] + b2[0], b2[1] - b1[0]);
                // Block (8..11, 8..11): dd = -(+) parts of P by row part p; k = -i (P - P^+).
                const double rv = __shfl_xor_sync(0xffffffffu, dd[0], 4);
                const double vv = df_flip(rv, psign) - dd[1];
                const double ww = __shfl_sync(0xffffffffu, vv, vsrc);
                kV = vv + df_flip(ww, psign);
              }
              // Re P = t1 + t2, Im P = t3 - t1 + t2; k = -i (P - P^+).
              double pr[2], pi[2], qr[2], qi[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                pr[e] = t1[e] + t2[e];
                pi[e] = (t3[e] - t1[e]) + t2[e];
                qr[e] = pr[e];
                qi[e] = pi[e];
              }
              transpose8(qr[0], qr[1]);
              transpose8(qi[0], qi[1]);
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const double kx = pi[e] + qi[e], ky = qr[e] - pr[e];
                sT_[kk][e].x = fma(wgt, kx, sT_[kk][e].x);
                sT_[kk][e].y = fma(wgt, ky, sT_[kk][e].y);
                xT[kk][e].x = fma(cn, kx, rT[kk][e].x);
                xT[kk][e].y = fma(cn, ky, rT[kk][e].y);
              }
              if constexpr (BIG) {
                sU[kk].x = fma(wgt, kU.x, sU[kk].x);
                sU[kk].y = fma(wgt, kU.y, sU[kk].y);
                sV_[kk] = fma(wgt, kV, sV_[kk]);
                xU[kk].x = fma(cn, kU.x, rU[kk].x);
                xU[kk].y = fma(cn, kU.y, rU[kk].y);
                xV[kk] = fma(cn, kV, rV[kk]);
              }
            }
          }
          // rho += dt/6 (k1 + 2 k2 + 2 k3 + k4) (src/solver.cpp:170-180); the elements i <= j staged for the
          // current.
#pragma unroll
          for (int kk = 0; kk < KPW; ++kk)
            if (kval[kk]) {
              double* R = RHO + (size_t)(w * KPW + kk) * rhos;
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                rT[kk][e].x = fma(prefac, sT_[kk][e].x, rT[kk][e].x);
                rT[kk][e].y = fma(prefac, sT_[kk][e].y, rT[kk][e].y);
                if (sT[e] == 0u && eT[e] != ze) *reinterpret_cast<double2*>(R + 2 * eT[e]) = rT[kk][e];
              }
              if constexpr (BIG) {
                rU[kk].x = fma(prefac, sU[kk].x, rU[kk].x);
                rU[kk].y = fma(prefac, sU[kk].y, rU[kk].y);
                rV[kk] = fma(prefac, sV_[kk], rV[kk]);
                if (eU != ze) *reinterpret_cast<double2*>(R + 2 * eU) = rU[kk];
                if (eV != ze && c4 <= h) R[2 * eV + p] = rV[kk];
              }
            }
        }
        df_cp_wait();
        __syncthreads();
        // The current of this step beside the H of the next.
        if (w >= NOW) {
          current(ti, w - NOW);
        } else if (ti + 1 < step1) {
          outer(ti + 1, false, w, NOW);
        }
        __syncthreads();
      }
      flush(step1 - 1);
#pragma unroll
      for (int kk = 0; kk < KPW; ++kk)
        if (kval[kk]) {
          double2* dst = rho + ((size_t)(m10 + w * KPW + kk) * t.N2 + m2) * nw2;
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (eT[e] != ze) dst[g * nw + 2 * c4 + e] = rT[kk][e];
          if constexpr (BIG) {
            if (eU != ze) {
              dst[g * nw + 8 + c4] = rU[kk];
              dst[(8 + c4) * nw + g] = make_double2(rU[kk].x, -rU[kk].y);
            }
            if (eV != ze) reinterpret_cast<double*>(dst + (8 + c4) * nw + 8 + h)[p] = rV[kk];
          }
        }
    }
}

using DfKernel = void (*)(SolveTables, DfData, int, double2*, double2*);
template <bool BIG, bool KM>
DfKernel df_kernel_nax(int nax) {
  return nax == 1   ? propagate_dfrag_kernel<BIG, 1, KM>
         : nax == 2 ? propagate_dfrag_kernel<BIG, 2, KM>
                    : propagate_dfrag_kernel<BIG, 3, KM>;
}
DfKernel df_kernel(const SolveTables& t) {
  if (t.nw > 8) return t.kmode ? df_kernel_nax<true, true>(t.nax) : df_kernel_nax<true, false>(t.nax);
  return t.kmode ? df_kernel_nax<false, true>(t.nax) : df_kernel_nax<false, false>(t.nax);
}
int df_kpc(const SolveTables& t) { return t.nw > 8 ? 8 : 16; }
DfLayout df_layout(const SolveTables& t) {
  return DfLayout(t.nw, t.nax, t.nj, df_kpc(t), t.kmode != 0, df_current_warps(t.nw > 8, t.kmode != 0));
}

}  // namespace

// The solves this kernel takes: 3..12 orbitals, a Hermitian placement whose box is symmetric about zero, at
// most 7 cells high (two k-steps) and 63 wide, at least one field axis and at most two current axes.  Over that whole range it is
// faster than the element-group kernel, which keeps the others: 512 steps of a 60 x 60 grid, two axes,
// element groups / this kernel: 3 orbitals 4.7 / 2.5 ms, 4: 4.2 / 2.6, 5: 9.2 / 2.7, 6: 9.8 / 2.9, 8: 21.8 / 3.3,
// 9: 27.3 / 7.1, 10: 34.4 / 7.4, 12: 28.8 / 8.2 (k-space solver 3: 7.8 / 2.7, 8: 38.4 / 3.7, 12: 36.2 / 11.1; 20 x 20,
// 3 orbitals: 4.0 / 1.6).  HHG_DFRAG=0 turns it off (measurements).
bool plan_dfrag(const SolveTables& t, int sm_count, LaunchShape* out) {
  if (const char* env = std::getenv("HHG_DFRAG"))
    if (env[0] == '0') return false;
  if (t.nw < 3 || t.nw > 12 || t.nax < 1 || t.nj > kDfNj || !t.hermitian) return false;
  if (t.b1n > 7 || t.b1n % 2 == 0 || t.b1lo != -(t.b1n - 1) / 2) return false;
  if (t.b2n > 63 || t.b2n % 2 == 0 || t.b2lo != -(t.b2n - 1) / 2) return false;
  const DfLayout L = df_layout(t);
  DfKernel kern = df_kernel(t);
  if (!allow_shared_memory(kern, L.bytes)) return false;
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kDfThreads, L.bytes);
  if (occ < 1) return false;
  const int kpc = df_kpc(t), rows = t.row1 - t.row0;
  const long slots = (long)occ * sm_count, ntiles = (long)t.N2 * ((rows + kpc - 1) / kpc);
  out->kernel = 5;
  out->kmode = t.kmode;
  out->ept = 1;
  out->variant = -1;
  out->k_per_cta = kpc;
  out->group = 32;
  out->threads = kDfThreads;
  out->ntiles = (int)ntiles;
  out->ctas = (int)(ntiles < slots ? ntiles : slots);
  out->vctas = out->ctas;
  out->box_sm = out->win_sm = 0;
  out->smem = L.bytes;
  out->pre_chunk = std::min(kDfChunk, t.nt);
  const size_t pts = t.kmode ? 2 * (size_t)out->pre_chunk + 1 : (size_t)out->pre_chunk;
  out->pre_bytes = 8 * t.N2 * (pts * L.gpt + (t.kmode ? 1 : pts) * L.wpt);
  return true;
}

int launch_dfrag(const SolveTables& t, const GroupTables& gt, const LaunchShape& s, double2* rho, double2* Jpart,
                 cudaStream_t stream) {
  if (!gt.pre || s.pre_chunk <= 0)
    throw std::runtime_error("FP64 fragment kernel launch: needs its precomputed-sum scratch (GroupTables::pre)");
  const DfLayout L = df_layout(t);
  const size_t pts_max = t.kmode ? 2 * (size_t)s.pre_chunk + 1 : (size_t)s.pre_chunk;
  double* GB = static_cast<double*>(gt.pre);
  double* CW = GB + pts_max * t.N2 * L.gpt;
  const DfData d = {gt.Xbox64, gt.Xwin64, gt.P64, gt.T1_64, gt.T2_64, GB, CW};
  DfKernel kern = df_kernel(t);
  allow_shared_memory(kern, s.smem);
  int launches = 0;
  for (int c0 = t.step0; c0 < t.step1; c0 += s.pre_chunk) {
    SolveTables tc = t;
    tc.step0 = c0;
    tc.step1 = std::min(c0 + s.pre_chunk, t.step1);
    const int npts = t.kmode ? 2 * (tc.step1 - c0) + 1 : tc.step1 - c0;
    dfrag_sums_kernel<<<dim3(t.N2, (npts + kDfSumPts - 1) / kDfSumPts), kDfSumThreads, 0, stream>>>(tc, d, L.nt, GB, CW, npts);
    kern<<<s.ctas, s.threads, s.smem, stream>>>(tc, d, s.vctas, rho, Jpart);
    launches += 2;
  }
  return launches;
}

}  // namespace hhg
