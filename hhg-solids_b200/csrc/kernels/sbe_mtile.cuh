// Mixed-form propagation for 6, 11 and 12 orbitals in 3 x 3 register tiles, half a warp per k-point of 11 and 12
// (included by sbe_group.cu, inside its anonymous namespace: it uses GroupData, the precomputed inner
// sums of group_sums_kernel and the helpers defined there).
//
// Same propagation as group_vctas in its mixed form (k-space-resident RK4 of the reference's
// src/solver.cpp:86-181, 1428-1726, and the windowed current of src/observable.cpp:16-30), for solves
// whose cell box is the Hermitian-halved 7x7 one and whose inner Wannier sums come precomputed per
// column and step (both solvers).
//
// Layout.  A CTA holds KPC consecutive k-points (rows m1) of one k-grid column; the k-point's matrices
// are padded to a 12 x 12 frame (11 and 12 orbitals; it takes 9..12: 16 lanes, half a warp, per k-point, 8 per CTA)
// or a 6 x 6 one (6 orbitals; it takes 4..6: 4 lanes per k-point, 32 per CTA), lane s owning its 3 x 3 tile (rows
// 3 (s / T) .. +2, columns 3 (s % T) .. +2, T tiles per frame row).  Each lane keeps its tile of the state rho and of the RK4
// sum in FP64 registers; the outer Wannier sums H0(k), r_a(k) of its elements (Geom::SHARE: which) give
// H = H0 + E.r at the step's field samples, the later ones kept in FP32 registers for their stages.
// Per stage:
//  * H = H0 + E.r goes to shared memory, transposed (H(i, j) at [j][i]), X = rho + c k
//    (FP32) is already there;
//  * the lane forms its tile of P = H X in FP32 from rows l of both arrays (three H and three X
//    values per l: 36 FMA per 6 loads, every load a broadcast to the lanes of its tile row or
//    column);
//  * k = -i (P - P^+) takes P^+ from the lane of the transposed tile, by shuffles (Geom::SHFL) or through the
//    place of X in shared memory;
//  * the RK4 sum and the next stage's X are formed in FP64 (X stored as FP32).
// Only the k-point's lanes (within one warp) exchange data, so the stages need __syncwarp only; the CTA meets twice
// per step for the current (its FP64 window rows copied in during the step, then the FP64 state staged
// for it) and once at its end (the next step's inner sums, copied in with cp.async meanwhile, and the
// current partials).  The current is FP64: summed over the CTA's k-points on the FP64 tensor cores, then
// contracted with the window rows.
//
// What bounds it: shared-memory wavefronts and instruction issue, together with the latency of a stage at 12 warps per
// SM; no pipe alone (packing the outer sums' multiply-adds as well, half their instructions, is 2 % slower).  So the
// arrays are laid out for the fewest wavefronts.  Measured on B200 (1965 MHz), 150 x 150, 256 steps, before and with
// rows of 12 in the inner sums, row factors formed once per CTA and k-points RS apart: 11 orbitals 17.27 and 16.34 ms,
// two field axes 19.98 and 18.10; 12 orbitals, 100 x 100, 7.98 and 7.75; k-space solver, 100 x 100, with shared outer
// sums as well: 11 orbitals 10.28 and 8.53, two axes 15.55 and 12.07; 12 orbitals 11.54 and 11.13, 13.43 and 12.90.
//
// Precision: as the element-group kernel's mixed form (complex-FP32 Wannier sums and commutator
// products, FP64 state, RK4 accumulation, window velocity and k-sum).

namespace mtile {

// Two FP32 values in one 64-bit register pair, and d = a b + c on both (fma.rn.f32x2: each half rounds as fmaf).
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// Waits until at most one committed group of this thread's cp.async copies is still in flight.
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <int NW, int NAX, int NJ, int KPC, bool KM = false>
struct Geom {
  static constexpr int NW2 = NW * NW;
  static constexpr int NMAT = 1 + NAX;
  static constexpr int NBROWS = NMAT * 4;   // halved 7 x 7 box: inner-sum rows n1 = 0..3 per matrix
  static constexpr int NWROWS = NJ * 4;     // window rows
  // The frame: 12 x 12 (9..12 orbitals) or 6 x 6 (4..6), in 3 x 3 tiles, one lane per tile; a CTA of
  // 128 threads holds KPC = 128 / (lanes per k-point) k-points (8 or 32).
  static constexpr int NWP = NW > 6 ? 12 : 6;
  static constexpr int TD = NWP / 3;        // tiles per frame row
  static constexpr int LPK = TD * TD;       // lanes per k-point
  static constexpr int NWARP = KPC * LPK / 32;
  // Inner-sum slots: this step's point and the next one's (real-space solver); the k-space solver's
  // points t + dt/2 and t + dt of this step and of the next, in a ring of four (point p in (p + 3) % 4).
  static constexpr int NGS = KM ? 4 : 2;
  static constexpr int NTHR = KPC * LPK;
  static constexpr int MS = NWP;            // row stride (float2) of a padded matrix
  static constexpr int KS = NWP * NWP + 1;  // float2 per k-point matrix: the odd 8-byte unit puts a
                                            // warp's k-points in different banks
  // Who forms which outer sums.  Real-space solver and the 6 x 6 frame: each lane its own tile.  k-space solver, 12 x
  // 12 frame, which forms them twice a step (SHARE): the 32 lanes of two neighbouring k-points take four elements of
  // both each, and where those are not all (12 orbitals) one more of one of them, so that a load serves two k-points
  // (8.5 against 9.2 ms; formed once a step it is the slower form, 17.1 against 16.3: two sets of factors in registers).
  static constexpr bool SHARE = KM && NWP == 12;
  static constexpr int PL = 2 * LPK;
  static constexpr bool SINGLE = !SHARE || NW2 > 4 * PL;
  static constexpr int NOUT = SINGLE ? 9 : 8;  // elements of H that a lane forms
  static constexpr int HMS = SINGLE ? MS : NWP + 1, HKS = SINGLE ? KS : NWP * HMS + 1;  // strides of H
  // P^+ by shuffles between the lanes of transposed tiles, which saves half the exchange's wavefronts and two of four
  // warp barriers per stage: 6 orbitals 9.51 -> 9.06 ms (150 x 150, 512 steps), k-space solver 2.87 -> 2.68, 11 orbitals
  // 1 %.  12 orbitals keep it in shared memory (from 1 % faster to 2 % slower with shuffles).
  static constexpr bool SHFL = NW < 12;
  static constexpr bool STAGED = NWP == 12;    // row factors formed once per CTA and point
  // Row stride and size of an inner-sum matrix: rows of 12 keep the tiles of a half warp in different banks, also
  // transposed (with rows of 11 three pairs of the 16 collide).
  static constexpr int GR = SHARE ? NW : NWP, GE = GR * NW;
  static constexpr size_t HS = 0;                                     // [KPC][HKS] float2: H, transposed
  static constexpr size_t XP = HS + (size_t)KPC * HKS * 8;            // [KPC][KS] float2: X, then P
  // The current's state lies over the H and X area, k-points RS double2 apart: 2 or 6 above a multiple of 8 keeps the
  // (k-point, element) pairs of its product's operand in different banks (12 x 12 frame; 6 x 6: 1 % slower with it).
  static constexpr int RS = NWP == 12 ? NW2 + (6 - NW2 % 4) % 4 : NW2;
  static constexpr size_t HXB = XP + (size_t)KPC * KS * 8, RSB = (size_t)KPC * RS * 16;
  static constexpr size_t GS = ((HXB > RSB ? HXB : RSB) + 15) / 16 * 16;  // [NGS][NBROWS][GE] float2
  static constexpr size_t GWS = GS + NGS * (size_t)NBROWS * GE * 8;  // [NWROWS][NW2] double2: one step's
                                                                      // (k-space solver: the column's)
  static constexpr size_t TW1 = GWS + (size_t)NWROWS * NW2 * 16;      // [KPC][8] float2: box rows q = 0..6
  static constexpr size_t P1S = TW1 + (size_t)KPC * 8 * 8;            // [NGS][KPC][8] float2: those times a point's phases
  static constexpr size_t WTW1 = P1S + (STAGED ? (size_t)NGS * KPC * 8 * 8 : 0);  // [KPC][4] double2: window rows
  static constexpr size_t SJ = WTW1 + (size_t)KPC * 4 * 16;           // [2][kJRing][NWARP][2 NJ] double
  static constexpr size_t BYTES = SJ + 2 * (size_t)kJRing * NWARP * 2 * NJ * 8;
  static_assert((NW > 8 && NW <= 12) || (NW >= 4 && NW <= 6), "3 x 3 tiles of a 12 x 12 or 6 x 6 frame");
  static_assert(!SHARE || (NW2 <= 4 * PL + PL / 2 && (!SINGLE || NW == NWP)), "the lanes' elements cover the matrix once");
  static_assert(KPC * LPK == 128, "128 threads per CTA");
  static_assert((NBROWS * GE * 8) % 16 == 0, "16-byte copies of the inner sums");
  static_assert(KPC % 4 == 0, "the current's product takes the CTA's k-points as its K dimension (k-steps of 4)");
};

// 128 threads per CTA run three CTAs per SM (at most 168 registers per thread): 12 warps per SM, against
// 8 for 16 k-points of 11 orbitals per CTA at 218 registers (C2: 324 against 416 ms per solve).
// KM: the reference's k-space solver (src/solver_kspace.cpp:167-270): the stages see H at points
// 2 ti (t), 2 ti + 1 (t + dt/2) and 2 ti + 2 (t + dt) of the interpolation tables; the outer sums of
// 2 ti + 2 stay in registers for the next step's first stage, and the window has no phase.
// PACK: the product in packed pairs; else in scalar operations (the planner's rule says where each is the faster).
template <int NW, int NAX, int NJ, int KPC, bool KM, bool PACK>
__global__ void __launch_bounds__(128, 3)
    propagate_mtile_kernel(SolveTables t, GroupData<float> d, int vctas, double2* rho, double2* Jpart) {
  using FG = Geom<NW, NAX, NJ, KPC, KM>;
  constexpr int NW2 = FG::NW2, NMAT = FG::NMAT, NWARP = FG::NWARP, NTHR = FG::NTHR, MS = FG::MS, KS = FG::KS;
  constexpr int NOUT = FG::NOUT, HMS = FG::HMS, HKS = FG::HKS;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* HS = reinterpret_cast<float2*>(smraw + FG::HS);
  float2* XPb = reinterpret_cast<float2*>(smraw + FG::XP);
  float2* GS = reinterpret_cast<float2*>(smraw + FG::GS);
  double2* GWS = reinterpret_cast<double2*>(smraw + FG::GWS);
  float2* TW1 = reinterpret_cast<float2*>(smraw + FG::TW1);
  float2* P1S = reinterpret_cast<float2*>(smraw + FG::P1S);
  double2* WTW1 = reinterpret_cast<double2*>(smraw + FG::WTW1);
  double* SJ = reinterpret_cast<double*>(smraw + FG::SJ);

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kp = tid / FG::LPK, sub = tid % FG::LPK, i0 = 3 * (sub / FG::TD), j0 = 3 * (sub % FG::TD);
  const int rows = t.row1 - t.row0, bpc = (rows + KPC - 1) / KPC, ntiles = t.N2 * bpc;
  const int step0 = t.step0, step1 = t.step1, npw = 2 * t.np + 1;
  const double dt = t.dt, prefac = 0.1666666666666 * dt;
  constexpr size_t gbuf = (size_t)FG::NBROWS * FG::GE, wbuf = (size_t)FG::NWROWS * NW2;
  const int lt = lane - sub + sub % FG::TD * FG::TD + sub / FG::TD;  // the lane of the transposed tile
  float2* Hk = HS + kp * HKS;
  float2* Xk = XPb + kp * KS;
  const float2 fzero = make_float2(0.f, 0.f);
  const double2 dzero = make_double2(0.0, 0.0);
  // Tile slot u = 3 a + b is element (i0 + a, j0 + b).  On the padding (row or column >= NW) it is no element: whatever
  // H's unwritten padding leaves there reaches no slot of an element.
  auto valid = [&](int u) { return i0 + u / 3 < NW && j0 + u % 3 < NW; };
  auto own = [&](int u) { return (i0 + u / 3) * MS + j0 + u % 3; };   // (i, j) in X, P
  auto tra = [&](int u) { return (j0 + u % 3) * MS + i0 + u / 3; };   // (j, i): H, P^+
  // Elements of H formed by this lane (o = 0..NOUT - 1) and their way into the transposed H.  SHARE: o = 2 s + h is
  // slot s of k-point kpA + h, o = 8 slot 4 of kpB; el[s] packs the slot's (i, j): its index, that of (j, i), and the
  // place in H.  Slots are consecutive elements per warp (11 orbitals) or half a 3 x 3 tile per lane (12, whose even
  // rows would put consecutive (j, i) into the same banks).
  const int psub = tid % FG::PL, kpA = tid / FG::PL * 2, kpB = kpA + psub / FG::LPK;
  int el[5];
  if constexpr (FG::SHARE) {
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      int i, j;
      if constexpr (FG::SINGLE) {
        const int tl = psub % FG::LPK, u = s < 4 ? 4 * (psub / FG::LPK) + s : 8;
        i = 3 * (tl / FG::TD) + u / 3, j = 3 * (tl % FG::TD) + u % 3;
      } else {
        const int e = min(s * FG::PL + psub, NW2 - 1);  // lanes past the end form the last element once more
        i = e / NW, j = e % NW;
      }
      el[s] = (i * FG::GR + j) | (j * FG::GR + i) << 8 | (j * HMS + i) << 16;
    }
  }
  auto store_h = [&](int o, float2 h) {
    if constexpr (FG::SHARE)
      HS[(o == 8 ? kpB : kpA + (o & 1)) * HKS + (el[o >> 1] >> 16)] = h;
    else
      Hk[tra(o)] = h;
  };

  for (int v = blockIdx.x; v < vctas; v += gridDim.x)
    for (int tile = v; tile < ntiles; tile += vctas) {
      const int m2 = tile / bpc, m10 = t.row0 + (tile % bpc) * KPC;
      const int nown = min(KPC, t.row1 - m10);
      const bool kval = kp < nown;

      // Inner sums of point p into slot `slot`, and window rows of point p (16-byte asynchronous copies).
      auto fetch_sums = [&](int p, int slot) {
        const size_t blk = (size_t)(p - (KM ? 2 * step0 : step0)) * t.N2 + m2;
        const char* src = reinterpret_cast<const char*>(d.Gpre + blk * gbuf);
        char* dst = reinterpret_cast<char*>(GS + (size_t)slot * gbuf);
        constexpr int nA = (int)(gbuf * 8 / 16);
        for (int idx = tid; idx < nA; idx += NTHR) cp_async16(dst + (size_t)idx * 16, src + (size_t)idx * 16);
      };
      auto fetch_window = [&](int p) {
        const double2* wsrc = d.GWpre + ((KM ? 0 : (size_t)(p - step0) * t.N2) + m2) * wbuf;
        for (int idx = tid; idx < (int)wbuf; idx += NTHR) cp_async16(GWS + idx, wsrc + idx);
      };
      // The warps' current partials of the ring half ending at step ti_end, into this virtual CTA's row.
      auto flush = [&](int ti_end) {
        const int slot = (ti_end / kJRing) & 1, s = ti_end % kJRing;
        const int ti0 = max(ti_end - s, step0), nsteps = ti_end - ti0 + 1;
        const double* half = SJ + ((size_t)slot * kJRing + (ti0 % kJRing)) * NWARP * 2 * NJ;
        for (int idx = tid; idx < nsteps * NJ; idx += NTHR) {
          const int ss = idx / NJ, a = idx % NJ;
          double re = 0.0, im = 0.0;
          for (int ww = 0; ww < NWARP; ++ww) {
            re += half[(ss * NWARP + ww) * 2 * NJ + 2 * a];
            im += half[(ss * NWARP + ww) * 2 * NJ + 2 * a + 1];
          }
          const int ja = a == 0 ? t.j_id[0] : (a == 1 ? t.j_id[1] : t.j_id[2]);
          double2* dst = Jpart + ((size_t)v * t.nt + ti0 + ss) * 3 + ja;
          const double2 old = *dst;
          *dst = make_double2(old.x + re, old.y + im);
        }
      };

      for (int idx = tid; idx < KPC * 8; idx += NTHR) {
        const int m = idx / 8, q = idx % 8, m1 = min(m10 + m, t.row1 - 1);
        TW1[idx] = q < 7 ? d.T1[wrap_mod((long long)m1 * (t.b1lo + q), t.N1)] : fzero;
      }
      for (int idx = tid; idx < KPC * 4; idx += NTHR) {
        const int m = idx / 4, q = idx % 4, m1 = min(m10 + m, t.row1 - 1);
        WTW1[idx] = d.T1d[wrap_mod((long long)m1 * (q - 2), t.N1)];
      }
      // Row factors p1(k, q) of the CTA's k-points at point p into slot `slot`: the rows' twiddles times the phases.
      auto row_factors = [&](int p, int slot) {
        if constexpr (FG::STAGED) {
          const float2* P1 = d.P + (size_t)p * 2 * npw + t.np + t.b1lo;
          for (int idx = tid; idx < KPC * 8; idx += NTHR)
            if (idx % 8 < 7) P1S[(size_t)slot * KPC * 8 + idx] = mul(TW1[idx], P1[idx % 8]);
        }
      };
      // Outer sums of the lane's elements at point p from GS slot `slot`: for matrix mat (H0, then r_a),
      // sum_{q=0..6} p1(k, q) G'(q)_e with G'(q) = G(n1 = q - 3) for q >= 3 and G(3 - q)^+ below;
      // take(o, m) receives element o's NMAT sums.
      auto outer = [&](int p, int slot, auto&& take) {
        const float2* G = GS + (size_t)slot * gbuf;
        auto factors = [&](int k, float2 (&f)[7]) {
          const float2* P1 = d.P + (size_t)p * 2 * npw + t.np;
#pragma unroll
          for (int q = 0; q < 7; ++q)
            f[q] = FG::STAGED ? P1S[((size_t)slot * KPC + k) * 8 + q] : mul(TW1[k * 8 + q], P1[t.b1lo + q]);
        };
        auto add_pair = [](const float2 (&f)[7], int n, float2 g, float2 gt, float2 acc) {
          return fmac(f[3 - n], conjugate(gt), fmac(f[3 + n], g, acc));
        };
        if constexpr (FG::SHARE) {
          float2 fA[7], fB[7];
          factors(kpA, fA);
          factors(kpA + 1, fB);
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const float2 *Ge = G + (el[s] & 255), *Gt = G + (el[s] >> 8 & 255);
            float2 mA[NMAT], mB[NMAT];
#pragma unroll
            for (int mat = 0; mat < NMAT; ++mat) {
              const float2 g0 = Ge[mat * 4 * FG::GE];
              mA[mat] = mul(fA[3], g0);
              mB[mat] = mul(fB[3], g0);
#pragma unroll
              for (int n = 1; n < 4; ++n) {
                const float2 g = Ge[(mat * 4 + n) * FG::GE], gt = Gt[(mat * 4 + n) * FG::GE];
                mA[mat] = add_pair(fA, n, g, gt, mA[mat]);
                mB[mat] = add_pair(fB, n, g, gt, mB[mat]);
              }
            }
            take(2 * s, mA);
            take(2 * s + 1, mB);
          }
          if constexpr (FG::SINGLE) {
            const float2 *Ge = G + (el[4] & 255), *Gt = G + (el[4] >> 8 & 255);
            float2 m[NMAT];
#pragma unroll
            for (int q = 0; q < 7; ++q) fA[q] = kpB == kpA ? fA[q] : fB[q];
#pragma unroll
            for (int mat = 0; mat < NMAT; ++mat) {
              m[mat] = mul(fA[3], Ge[mat * 4 * FG::GE]);
#pragma unroll
              for (int n = 1; n < 4; ++n)
                m[mat] = add_pair(fA, n, Ge[(mat * 4 + n) * FG::GE], Gt[(mat * 4 + n) * FG::GE], m[mat]);
            }
            take(8, m);
          }
        } else {
          float2 f[7];
          factors(kp, f);
#pragma unroll
          for (int u = 0; u < 9; ++u) {
            float2 m[NMAT];
#pragma unroll
            for (int mat = 0; mat < NMAT; ++mat) {
              m[mat] = fzero;
              if (valid(u)) {
                const int i = i0 + u / 3, j = j0 + u % 3, e = i * FG::GR + j, eT = j * FG::GR + i;
                const float2* Gm = G + (size_t)mat * 4 * FG::GE;
                m[mat] = mul(f[3], Gm[e]);
#pragma unroll
                for (int n = 1; n < 4; ++n) m[mat] = add_pair(f, n, Gm[n * FG::GE + e], Gm[n * FG::GE + eT], m[mat]);
              }
            }
            take(u, m);
          }
        }
      };
      // The field samples of step ts (t, t + dt/2, t + dt) on the active axes, and H = H0 + E.r.
      auto fields = [&](int ts, float (&ea)[3][NAX]) {
        const double* es = t.es + (size_t)ts * 9;
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
          for (int a = 0; a < NAX; ++a) ea[f][a] = (float)es[f * 3 + t.ax_id[a]];
      };
      auto field_h = [&](const float2 (&m)[NMAT], const float (&e)[NAX]) {
        float2 h = m[0];
#pragma unroll
        for (int a = 0; a < NAX; ++a) {
          h.x = fmaf(e[a], m[1 + a].x, h.x);
          h.y = fmaf(e[a], m[1 + a].y, h.y);
        }
        return h;
      };
      // H of the lane's elements at the step's later stages (registers): real-space solver, at t + dt/2 and t + dt
      // (H at t goes to shared memory as the sums are formed); k-space solver, the next step's H at t.
      float2 Hn[KM ? 1 : 2][NOUT];
      auto gslot = [&](int p) { return KM ? (p + 3) & 3 : p & 1; };

      if constexpr (KM) {
        fetch_sums(2 * step0, gslot(2 * step0));
        fetch_window(0);  // the column's window rows, the same for every step
      } else {
        fetch_sums(step0, gslot(step0));
      }
      cp_async_commit();
      // This lane's tile of the state (FP64 registers for the whole tile).
      const size_t kg = ((size_t)(m10 + (kval ? kp : 0)) * t.N2 + m2) * NW2;
      double2 r[9];
#pragma unroll
      for (int u = 0; u < 9; ++u) r[u] = (kval && valid(u)) ? rho[kg + (i0 + u / 3) * NW + j0 + u % 3] : dzero;
      if constexpr (FG::STAGED) __syncthreads();
      row_factors(KM ? 2 * step0 : step0, gslot(KM ? 2 * step0 : step0));
      cp_async_wait_all();
      __syncthreads();
      if constexpr (KM) {
        // The chunk's first point t (then carried from step to step), and the first step's other two.
        {
          float ea[3][NAX];
          fields(step0, ea);
          outer(2 * step0, gslot(2 * step0), [&](int o, const float2 (&m)[NMAT]) { Hn[0][o] = field_h(m, ea[0]); });
        }
        fetch_sums(2 * step0 + 1, gslot(2 * step0 + 1));
        fetch_sums(2 * step0 + 2, gslot(2 * step0 + 2));
        cp_async_commit();
        row_factors(2 * step0 + 1, gslot(2 * step0 + 1));
        row_factors(2 * step0 + 2, gslot(2 * step0 + 2));
        cp_async_wait_all();
        __syncthreads();
      }

      for (int ti = step0; ti < step1; ++ti) {
        const int buf = ti & 1;
        if (ti > step0 && (ti - 1) % kJRing == kJRing - 1) flush(ti - 1);
        if constexpr (KM) {
          // The next step's points t + dt/2 and t + dt, into the slots of this step's t and of the
          // previous step's t + dt/2, whose last readers finished before the barrier that ended it.
          if (ti + 1 < step1) {
            fetch_sums(2 * ti + 3, gslot(2 * ti + 3));
            fetch_sums(2 * ti + 4, gslot(2 * ti + 4));
            row_factors(2 * ti + 3, gslot(2 * ti + 3));
            row_factors(2 * ti + 4, gslot(2 * ti + 4));
          }
          cp_async_commit();
        } else {
          // This step's window rows (read by the current at its end), then the next step's inner sums
          // into the other slot: both buffers' last readers finished before the barrier that ended the
          // previous step.  Two groups, so that the current can wait for the first alone.
          fetch_window(ti);
          cp_async_commit();
          if (ti + 1 < step1) {
            fetch_sums(ti + 1, gslot(ti + 1));
            row_factors(ti + 1, gslot(ti + 1));
          }
          cp_async_commit();
          // (1) Outer sums at the step's point: H at t into shared memory (the area's last readers, the
          //     previous step's current, finished before the barrier), at t + dt/2 and t + dt kept.
          float ea[3][NAX];
          fields(ti, ea);
          outer(ti, buf, [&](int o, const float2 (&m)[NMAT]) {
            store_h(o, field_h(m, ea[0]));
            Hn[0][o] = field_h(m, ea[1]);
            Hn[1][o] = field_h(m, ea[2]);
          });
        }
        // (2) RK4 stages (src/solver.cpp:157-180), fields at t, t+dt/2, t+dt/2, t+dt; X = rho for the first
        //     (the area held the previous step's FP64 state for the current).
#pragma unroll
        for (int u = 0; u < 9; ++u) Xk[own(u)] = make_float2((float)r[u].x, (float)r[u].y);
        double2 S[9];
#pragma unroll 1
        for (int st = 0; st < 4; ++st) {
          // H of the stage (the third keeps the second's: same field and point).
          if constexpr (KM) {
            float ea[3][NAX];
            fields(ti, ea);
            if (st == 0) {
#pragma unroll
              for (int o = 0; o < NOUT; ++o) store_h(o, Hn[0][o]);
            } else if (st == 1) {
              outer(2 * ti + 1, gslot(2 * ti + 1), [&](int o, const float2 (&m)[NMAT]) { store_h(o, field_h(m, ea[1])); });
            } else if (st == 3) {
              // the point t + dt: this stage's H, and the next step's H at t (its first field sample)
              float en[3][NAX];
              fields(ti + 1 < step1 ? ti + 1 : ti, en);
              outer(2 * ti + 2, gslot(2 * ti + 2), [&](int o, const float2 (&m)[NMAT]) {
                store_h(o, field_h(m, ea[2]));
                Hn[0][o] = field_h(m, en[0]);
              });
            }
          } else {
            if (st == 1) {
#pragma unroll
              for (int o = 0; o < NOUT; ++o) store_h(o, Hn[0][o]);
            } else if (st == 3) {
#pragma unroll
              for (int o = 0; o < NOUT; ++o) store_h(o, Hn[1][o]);
            }
          }
          __syncwarp();
          // P = H X on the tile: P(i, j) = sum_l H(i, l) X(l, j), H(i, l) from row l of the transposed H.
          float2 P[9];
          if constexpr (PACK) {
            // Each complex multiply-add is two packed ones, h.x (x, y) then h.y (-y, x): the roundings and their
            // order of four scalar ones.
            F2 acc[9];
#pragma unroll
            for (int u = 0; u < 9; ++u) acc[u] = pack2(0.f, 0.f);
#pragma unroll
            for (int l = 0; l < NW; ++l) {
              const float2* hr = Hk + l * HMS + i0;
              const float2* xr = Xk + l * MS + j0;
              F2 xa[3], xb[3];
#pragma unroll
              for (int c = 0; c < 3; ++c) {
                const float2 q = xr[c];
                xa[c] = pack2(q.x, q.y);
                xb[c] = pack2(-q.y, q.x);
              }
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                const float2 h = hr[a];
                const F2 hx = pack2(h.x, h.x), hy = pack2(h.y, h.y);
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[3 * a + c] = fma2(hy, xb[c], fma2(hx, xa[c], acc[3 * a + c]));
              }
            }
#pragma unroll
            for (int u = 0; u < 9; ++u) P[u] = unpack2(acc[u]);
          } else {
#pragma unroll
            for (int u = 0; u < 9; ++u) P[u] = fzero;
#pragma unroll
            for (int l = 0; l < NW; ++l) {
              const float2* hr = Hk + l * HMS + i0;
              const float2* xr = Xk + l * MS + j0;
              const float2 h[3] = {hr[0], hr[1], hr[2]}, x[3] = {xr[0], xr[1], xr[2]};
#pragma unroll
              for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) P[3 * a + c] = fmac(h[a], x[c], P[3 * a + c]);
            }
          }
          __syncwarp();  // every lane of the k-point has read X and H
          if constexpr (!FG::SHFL) {
#pragma unroll
            for (int u = 0; u < 9; ++u) Xk[own(u)] = P[u];
            __syncwarp();
          }
          const double wgt = (st == 0 || st == 3) ? 1.0 : 2.0;
          const double cn = (st == 2 ? 1.0 : 0.5) * dt;
          float2 xn[9];
#pragma unroll
          for (int u = 0; u < 9; ++u) {
            const int ut = 3 * (u % 3) + u / 3;  // P(j, i): this place of the transposed tile
            const float2 pt = FG::SHFL ? make_float2(__shfl_sync(0xffffffffu, P[ut].x, lt), __shfl_sync(0xffffffffu, P[ut].y, lt))
                                       : Xk[tra(u)];
            const float kx = P[u].y + pt.y, ky = -(P[u].x - pt.x);  // k = -i (P - P^+)
            if (st == 0) {
              S[u] = make_double2((double)kx, (double)ky);
            } else {
              S[u].x += wgt * (double)kx;
              S[u].y += wgt * (double)ky;
            }
            xn[u] = make_float2((float)(r[u].x + cn * (double)kx), (float)(r[u].y + cn * (double)ky));
          }
          if constexpr (!FG::SHFL) __syncwarp();  // every lane of the k-point has read P
          if (st < 3) {
#pragma unroll
            for (int u = 0; u < 9; ++u) Xk[own(u)] = xn[u];
          }
        }
        // rho += dt/6 (k1 + 2 k2 + 2 k3 + k4) (src/solver.cpp:170-180).
#pragma unroll
        for (int u = 0; u < 9; ++u) {
          r[u].x = r[u].x + prefac * S[u].x;
          r[u].y = r[u].y + prefac * S[u].y;
        }

        // (3) Current partials of step ti (FP64), summed over the CTA's k-points before the window:
        //     J_a = sum_{q,e} GW(a, q)_e R(q, e) with R(q, e) = sum_k wp(k, q) conj(rho_e(k)), the same sum
        //     as sum_k sum_e W_a(k)_e conj(rho_e(k)), W_a(k)_e = sum_q wp(k, q) GW(a, q)_e, in another order.
        //     R is a [4 window rows (of 8)] x [8 k-points] x [nw^2 elements] product on the FP64 tensor
        //     cores (three real m8n8k4 products per complex one) from the state staged in FP64 over the H
        //     and X area, which every k-point's stages have finished with at the barrier.
        if constexpr (!KM) cp_async_wait_one();  // this step's window rows
        __syncthreads();
        double2* RS = reinterpret_cast<double2*>(HS);  // [KPC][RS] double2
        if (kval) {
#pragma unroll
          for (int u = 0; u < 9; ++u)
            if (valid(u)) RS[kp * FG::RS + (i0 + u / 3) * NW + j0 + u % 3] = r[u];
        } else {
#pragma unroll
          for (int u = 0; u < 9; ++u)
            if (valid(u)) RS[kp * FG::RS + (i0 + u / 3) * NW + j0 + u % 3] = dzero;
        }
        __syncthreads();
        {
          const int g = lane >> 2, c4 = lane & 3;
          const double2* P1d = d.Pd + (size_t)ti * 2 * npw + t.np;
          // A[g][c] of k-step ks: wp(k-point 4 ks + c, window row g), rows 4..7 zero.
          constexpr int NKS = KPC / 4;
          double2 wa[NKS];
#pragma unroll
          for (int ks = 0; ks < NKS; ++ks)
            wa[ks] = g < 4 ? (KM ? WTW1[(4 * ks + c4) * 4 + g] : mul(WTW1[(4 * ks + c4) * 4 + g], P1d[g - 2])) : dzero;
          double re[3] = {0.0, 0.0, 0.0}, im[3] = {0.0, 0.0, 0.0};
          constexpr int NTR = (NW2 + 7) / 8;
#pragma unroll 1
          for (int nt = w; nt < NTR; nt += NWARP) {
            double t1[2] = {0.0, 0.0}, t2[2] = {0.0, 0.0}, t3[2] = {0.0, 0.0};
            const int eb = 8 * nt + g;  // B[c][g]: conj(rho_eb(k-point 4 ks + c))
#pragma unroll
            for (int ks = 0; ks < NKS; ++ks) {
              const double2 b = eb < NW2 ? RS[(4 * ks + c4) * FG::RS + eb] : dzero;
              dmma(t1, wa[ks].x, b.x);
              dmma(t2, wa[ks].y, -b.y);
              dmma(t3, wa[ks].x + wa[ks].y, b.x - b.y);
            }
            if (g < 4) {
#pragma unroll
              for (int jj = 0; jj < 2; ++jj) {
                const int e = 8 * nt + 2 * c4 + jj;  // R(g, e)
                if (e < NW2) {
                  const double rr = t1[jj] - t2[jj], ri = t3[jj] - t1[jj] - t2[jj];
#pragma unroll
                  for (int a = 0; a < NJ; ++a) {
                    const double2 gw = GWS[(a * 4 + g) * NW2 + e];
                    re[a] = fma(gw.x, rr, fma(-gw.y, ri, re[a]));
                    im[a] = fma(gw.x, ri, fma(gw.y, rr, im[a]));
                  }
                }
              }
            }
          }
          const int slot = (ti / kJRing) & 1, s = ti % kJRing;
          warp_store_current(re, im, NJ, lane, SJ + (((size_t)slot * kJRing + s) * NWARP + w) * 2 * NJ);
        }
        cp_async_wait_all();
        __syncthreads();
      }
      flush(step1 - 1);
      if (kval) {
#pragma unroll
        for (int u = 0; u < 9; ++u)
          if (valid(u)) rho[kg + (i0 + u / 3) * NW + j0 + u % 3] = r[u];
      }
      __syncthreads();
    }
}

}  // namespace mtile
