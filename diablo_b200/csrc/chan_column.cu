// The per-mode column stage of RK_CHAN_1 before REM_DIV: explicit terms, the
// Crank-Nicolson right-hand side and the CN solve of one field, for a tile of
// MT retained (kx, kz) modes and their whole y-columns.
//
// Reference steps it replaces, per mode instead of per physical column (the
// operators are linear and the same for every column, so they commute with
// the x-z transform):
//   RHS assembly     for/channel.f:88-167   CR = CU + zeta h CF - h grad P
//   explicit terms   for/channel.f:175-290  CF = -nu k^2 CU + Coriolis,
//                                           buoyancy, GRAV, DRHODX/Z + NL
//   CN explicit half for/channel.f:580-626  R += beta h CF + (nu h/2) d2/dy2 CU
//   CN solves        for/channel.f:771-1029 (THOMAS_*_MPI, for/mpi.f:630-866)
// REM_DIV_CHAN and the pressure update follow as their own launch (k_rd_col).
//
// A work item is (case, mode tile, field), one CTA; one thread per (mode,
// segment of K consecutive rows), the modes of a segment in neighbouring
// lanes.  The CN system of a field is the same for every
// mode, and its elimination (the substep's table: multipliers a, reciprocal
// pivots 1/b, f = -c/b) turns the solve into two first-order linear
// recurrences, forward g(j) = r(j) + a(j) g(j-1) and backward
// x(j) = e(j) + f(j) x(j+1) with e = g/b.  A linear recurrence splits exactly
// over segments: each thread runs its segment from a zero start, keeping the
// product of the coefficients; the (product, end value) of the segments, four at a time
// by shuffles and then quad by quad from shared memory, carry the
// segment ends through the column, and each thread adds carry x product to its rows.  The same
// algebra as THOMAS_FORWARD / THOMAS_BACKWARD, with the rounding of a different
// order of the same operations.  Segments and quads depend only on NY, so a
// mode's arithmetic does not depend on the tile width.
//
// Everything between the inputs and the post-CN field is in the thread's
// registers: it loads its rows of CU, NL (which the z-forward kernel left in the
// field's rhs array), CF_old and CP straight from global memory -- the lanes of a segment
// read neighbouring modes, whole sectors -- forms R, runs the recurrences and stores CF and the
// field, with one barrier per direction for the quads' totals.  Only the table
// and grid-factor rows, shared by every mode, go through shared memory (bulk
// copies on one mbarrier with a bounded wait).  CU is read-only in this kernel,
// so a field's right-hand side may read another field (rotation, buoyancy, GRAV,
// DRHODX/Z) without a race.  REM_DIV then reads the post-CN velocity from the rhs
// arrays and writes CU.  A scalar that no velocity right-hand side reads is
// written in place.
//
// It is bound by memory latency: 114 MB per launch at Re_tau = 180 in 41 us (1107 us
// at 512x257x384 with a scalar), 14 warps per SM at 128 registers.  Forms with the columns in shared memory (bulk
// tensor copies of CU and NL, CF and CP read beside them, the recurrences there with six
// barriers) took 52 us at 4 modes per CTA and 43 at 8 (1302 and 1042), and 51 with all four tiles staged and the
// recurrences in registers: the tiles allow two to four CTAs per SM, and each
// waits for its copies, computes and writes in turn.
//
// The same kernel serves one case (a one-case table) and the ensemble
// server's groups (a ragged work list over every member), so a case
// computes with the same machine code either way.
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "dg_internal.cuh"

namespace {

// Rows per segment: with 5 a thread's rows of all its inputs all but fit 128
// registers (Re_tau = 180: 41 us per launch; 43 with 4, 55 with 3; 54 with 7 and 65
// with 9, which spill); with 3 a short column takes less code, and time, to
// start up (64x33x16: 10.6 us, 14.6 with 5).
constexpr int SEG_K = 5, SEG_KS = 3, SEG_SHORT = 48;  // 3 up to 48 rows
constexpr int COL_MAX_THR = 512; // threads per CTA: MT x segments, rounded up to warps

struct ColConst {
  int NY, nf, nth, nkxp, JS, JE;
  int JSt[DG_MAX_TH], JEt[DG_MAX_TH];
  long ss;
  double nu, beta, nuv, i_ro, grav_x, grav_y, grav_z, px0, omega0, amp_omega0;
  int f_type;
  double ri[DG_MAX_TH], pr[DG_MAX_TH], drhodx[DG_MAX_TH], drhodz[DG_MAX_TH];
};

// Everything the column stage of one case needs, in device memory.
struct ColCase {
  ColConst C;
  const double *dscal, *tab, *kxv, *kzv, *rowc;
  const double2 *cp;
  const double2 *cu[3 + DG_MAX_TH], *nl[3 + DG_MAX_TH];
  double2 *cf[3 + DG_MAX_TH], *out[3 + DG_MAX_TH];  // out: the rhs arrays
  int *err;
  int nseg;
};

template <typename T>
__device__ __forceinline__ T pick(const T (&a)[DG_MAX_TH], int i) {
  T r = a[0];
#pragma unroll
  for (int k = 1; k < DG_MAX_TH; k++) r = (i == k) ? a[k] : r;
  return r;
}

__device__ __forceinline__ double2 z2() { return make_double2(0.0, 0.0); }

// rowc: per-row grid factors [8][LP] (LP = NY + 2 rounded up to even, so
// rows start on 16-byte boundaries for the bulk copies)
//   0 1/(DY(j+1) DYF(j))  1 1/(DY(j) DYF(j))       (GYF rows: U1, U3, TH)
//   2 1/(DYF(j) DY(j))    3 1/(DYF(j-1) DY(j))     (GY rows: U2)
//   4 1/DY(j)             5 DYF(j)                 (U2)
//   6 1/DYF(j)            7 REM_DIV upper diagonal

// The field's coefficients that do not change along the column, read from the
// case table once per CTA.  What other fields add to the explicit terms at row j
// is linear in them: sum_q w[q] X_q(j) over src[q] (U1, U3: rotation and RI
// GRAV_x/z TH; U2: RI GRAV_y TH, then interpolated to GY; a scalar: -DRHODX U1 - DRHODZ U3).
struct FieldCoef {
  double T3, T4, T5, aa, nu;
  double force;                     // T4 times the mean pressure gradient (U1)
  double w[1 + DG_MAX_TH];
  const double2 *src[1 + DG_MAX_TH];
  int nsrc;                         // 0: nothing couples
  int lo, hi;
};

__device__ __forceinline__ FieldCoef field_coef(const ColCase &cc, int rk_step, int f) {
  const ColConst &C = cc.C;
  FieldCoef k;
  const double h = cc.dscal[1 + rk_step];
  const double zeta = (rk_step == 2) ? -17.0 / 8.0 : (rk_step == 3) ? -5.0 / 4.0 : 0.0;
  const double bbar = (rk_step == 2) ? 25.0 / 8.0 : (rk_step == 3) ? 9.0 / 4.0 : 1.0;
  k.T3 = zeta * h;
  k.T4 = h;
  k.T5 = bbar * h;
  const int n = f - 3;
  const double ipr = (f >= 3) ? 1.0 / pick(C.pr, n) : 1.0;
  k.nu = (f >= 3) ? C.nu / pick(C.pr, n) : C.nu;
  k.aa = ipr * ((C.nu * h / 2.0) * C.nuv);
  k.force = 0.0;
  if (f == 0 && C.f_type == 1) k.force = k.T4 * C.px0;
  else if (f == 0 && C.f_type == 2)
    k.force = k.T4 * (C.px0 + C.amp_omega0 * cos(C.omega0 * cc.dscal[0]));
  k.nsrc = 0;
#pragma unroll
  for (int q = 0; q <= DG_MAX_TH; q++) {
    k.w[q] = 0.0;
    k.src[q] = cc.cu[0];
  }
  if (f >= 3) {
    k.w[0] = -pick(C.drhodx, n);
    k.w[1] = -pick(C.drhodz, n);
    k.src[1] = cc.cu[2];
    if (k.w[0] != 0.0 || k.w[1] != 0.0) k.nsrc = 2;
  } else {
    const double gr = (f == 0) ? C.grav_x : (f == 2) ? C.grav_z : C.grav_y;
    k.w[0] = (f == 0) ? C.i_ro : (f == 2) ? -C.i_ro : 0.0;
    k.src[0] = cc.cu[(f == 0) ? 2 : 0];
    if (k.w[0] != 0.0) k.nsrc = 1;
#pragma unroll
    for (int q = 0; q < DG_MAX_TH; q++) {
      if (q >= C.nth) break;
      k.w[1 + q] = C.ri[q] * gr;
      k.src[1 + q] = cc.cu[3 + q];
      if (k.w[1 + q] != 0.0) k.nsrc = 2 + q;
    }
  }
  if (f == 0 || f == 2) { k.lo = C.JS; k.hi = C.JE; }
  else if (f == 1) { k.lo = 2; k.hi = C.NY; }
  else { k.lo = pick(C.JSt, n); k.hi = pick(C.JEt, n); }
  return k;
}

// Launch-wide sizes: the largest item of the work list sets the layout.
struct ColLaunch {
  int lp;     // table row length (the largest case's NY + 2, rounded up to even)
  int nwork;  // work items (CTAs)
};

// Shared memory of one CTA: the CN table rows TB [5][lp] (a, 1/b, f = -c/b,
// kind, BC value); the field's grid factors RC [4][lp]; the totals of the quads (pairs) of
// segments for the two directions, end values TG [2][pairs][MT] double2 and products
// TP [2][pairs]; the mbarrier.
size_t col_smem_l(const ColLaunch &P, int mt, int thr) {
  const size_t pairs = thr / (2 * mt);
  return sizeof(double) * (9 * (size_t)P.lp + 2 * pairs * (2 * mt + 1)) + 16;
}

// What enters segment s of mode m from the segments before it (DIR = +1: rows
// above in index order; -1: from the last one back): the states (end value e, product p) of
// the segments compose as e2 + p2 X, (e, p) per segment, identity (0, 1) where a thread has no
// rows.  Segments go in pairs and quads (a fixed order, so that the result does not depend on
// the tile width): by shuffles inside a warp, which holds 32 / MT segments, the
// totals of the quads (of the pairs for MT = 16) in shared memory, then quad by quad.
template <int MT, int DIR>
__device__ __forceinline__ double2 carry(int s, int m, int nseg, double2 e, double p, double2 *TG,
                                         double *TP) {
  static_assert(MT <= 16, "the two segments of a pair share a warp");
  constexpr unsigned ALL = 0xffffffffu;
  const bool late = DIR > 0 ? (s & 1) : !(s & 1);      // second of its pair
  const bool late2 = DIR > 0 ? (s & 2) : !(s & 2);     // in the second pair of its quad
  const int lane = threadIdx.x & 31;
  // the pair
  const int src1 = lane ^ MT;
  const double2 o = make_double2(__shfl_sync(ALL, e.x, src1), __shfl_sync(ALL, e.y, src1));
  const double op = __shfl_sync(ALL, p, src1);
  double2 c = late ? o : z2();
  double pe = late ? op : 1.0;
  // the pair's total (right in its second segment)
  e = make_double2(e.x + p * o.x, e.y + p * o.y);
  p = p * op;
  if constexpr (MT <= 8) {
    // the first pair's total, from its second segment
    const int sw = lane / MT, q0 = sw & ~3;
    const int src2 = (q0 + (DIR > 0 ? 1 : 2)) * MT + m;
    const double2 t = make_double2(__shfl_sync(ALL, e.x, src2), __shfl_sync(ALL, e.y, src2));
    const double tp = __shfl_sync(ALL, p, src2);
    if (late2) {
      c = make_double2(c.x + pe * t.x, c.y + pe * t.y);
      pe = pe * tp;
    }
    if (late && late2) {
      TG[(s >> 2) * MT + m] = make_double2(e.x + p * t.x, e.y + p * t.y);
      if (m == 0) TP[s >> 2] = p * tp;
    }
  } else if (late) {
    TG[(s >> 1) * MT + m] = e;
    if (m == 0) TP[s >> 1] = p;
  }
  __syncthreads();
  const int quad = s >> 2, npair = blockDim.x / (2 * MT);
  if constexpr (MT > 8) {
    if (late2) {
      // the pair before this one (it may lie beyond the CTA's last thread)
      const int w = 2 * quad + (DIR > 0 ? 0 : 1);
      const double2 t = w < npair ? TG[w * MT + m] : z2();
      c = make_double2(c.x + pe * t.x, c.y + pe * t.y);
      pe = pe * (w < npair ? TP[w] : 1.0);
    }
  }
  // the quads before this one, four at a time (their loads ahead of the chain)
  const int nq = DIR > 0 ? quad : ((nseg - 1) >> 2) - quad;
  double2 X = z2();
  for (int w0 = 0; w0 < nq; w0 += 4) {
    double2 t[4];
    double tp[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int w = DIR > 0 ? w0 + i : ((nseg - 1) >> 2) - w0 - i;
      t[i] = z2();
      tp[i] = 1.0;
      if (w0 + i < nq) {
        if constexpr (MT <= 8) {
          t[i] = TG[w * MT + m];
          tp[i] = TP[w];
        } else {
          const int a = 2 * w + (DIR > 0 ? 0 : 1), b = 2 * w + (DIR > 0 ? 1 : 0);  // first, second
          const double2 ta = a < npair ? TG[a * MT + m] : z2(), tb = b < npair ? TG[b * MT + m] : z2();
          const double pa = a < npair ? TP[a] : 1.0, pb = b < npair ? TP[b] : 1.0;
          t[i] = make_double2(tb.x + pb * ta.x, tb.y + pb * ta.y);
          tp[i] = pb * pa;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) X = make_double2(t[i].x + tp[i] * X.x, t[i].y + tp[i] * X.y);
  }
  return make_double2(c.x + pe * X.x, c.y + pe * X.y);
}

// The column stage of field f (kind FK: 0 U1/U3, 1 U2, 2 scalar): explicit
// terms, CF, R and the CN solve of the thread's rows j0 .. j0+nr-1 of one mode,
// whose row 0 lies at offset mg of every field.
template <int MT, int K, int FK, bool CPL, typename Table>
__device__ __forceinline__ void col_rows(const FieldCoef &k, bool old_cf, int L, long ss, long mg,
                                         int j0, int nr, int nseg, bool mean, double Kh, double kk,
                                         int wlo,
                                         const double2 *cu, const double2 *nl,
                                         double2 *cff, const double2 *__restrict__ cpp,
                                         double2 *dst, const double *TB, const double *RC, int LP,
                                         double2 *TG, double *TP, Table table) {
  const int s = threadIdx.x / MT, m = threadIdx.x % MT;
  const int slots = blockDim.x / (2 * MT);
  const long o0 = (long)j0 * ss + mg;
  auto in = [&](int q) { return q < nr && j0 + q >= k.lo && j0 + q <= k.hi; };
  // ---- 1. R.  Every input row is on its way before the first is used, and
  // before the wait for the table rows.  A scalar written in place has dst == cu, and the
  // rows j0-1 and j0+K are other threads': plain loads there (the read-only path and
  // restrict want data that the launch does not write), all of them before the
  // first barrier of carry(), and every store to dst after its second.
  double2 r[K], p[K + 1], u[K + 2], v[K];  // CF_old, CP rows j0-1 .., CU rows j0-1 .., NL
#pragma unroll
  for (int q = 0; q < K; q++) r[q] = (old_cf && in(q)) ? cff[o0 + q * ss] : z2();
  if (FK < 2) {
#pragma unroll
    for (int q = 0; q < K; q++) p[q + 1] = in(q) ? __ldg(cpp + o0 + q * ss) : z2();
  }
  if (FK == 1) p[0] = (nr > 0 && j0 > 0) ? __ldg(cpp + o0 - ss) : z2();
#pragma unroll
  for (int q = 0; q < K + 2; q++) {
    const int j = j0 + q - 1;
    const bool have = nr > 0 && j >= 0 && j < L;
    if constexpr (FK == 2) u[q] = have ? cu[o0 + (q - 1) * ss] : z2();
    else u[q] = have ? __ldg(cu + o0 + (q - 1) * ss) : z2();
  }
#pragma unroll
  for (int q = 0; q < K; q++) v[q] = in(q) ? nl[o0 + q * ss] : z2();
  if (!table()) return;
#pragma unroll
  for (int q = 0; q < K; q++) {
    r[q].x *= k.T3;
    r[q].y *= k.T3;
    if (FK == 0) {
      // - h (i K P), Kh = h K
      r[q].x += Kh * p[q + 1].y;
      r[q].y -= Kh * p[q + 1].x;
    } else if (FK == 1 && in(q)) {
      const double c = k.T4 * RC[2 * LP + j0 + q];
      r[q].x -= c * (p[q + 1].x - p[q].x);
      r[q].y -= c * (p[q + 1].y - p[q].y);
    }
  }
  {
    // what other fields add (w X summed over the fields)
    auto others = [&](int q) -> double2 {
      double2 S = z2();
#pragma unroll
      for (int e = 0; e <= DG_MAX_TH; e++) {
        if (e >= k.nsrc) break;
        if (k.w[e] == 0.0) continue;
        const double2 x = __ldg(k.src[e] + o0 + q * ss);
        S.x += k.w[e] * x.x;
        S.y += k.w[e] * x.y;
      }
      return S;
    };
    double2 Sm = z2();
    if (CPL && FK == 1 && nr > 0 && j0 > 0) Sm = others(-1);
#pragma unroll
    for (int q = 0; q < K; q++) {
      double2 S = z2();
      if (CPL && q < nr) S = others(q);
      if (in(q)) {
        const int j = j0 + q;
        const double2 uc = u[q + 1];
        double2 fv = make_double2(-k.nu * kk * uc.x, -k.nu * kk * uc.y);
        if (FK == 1) {
          if (CPL && !mean) {
            const double dyfj = RC[3 * LP + j], dyfm = RC[3 * LP + j - 1];
            const double bw2 = 0.5 * RC[2 * LP + j];
            fv.x += bw2 * (S.x * dyfm + Sm.x * dyfj);
            fv.y += bw2 * (S.y * dyfm + Sm.y * dyfj);
          }
        } else if (CPL) {
          fv.x += S.x;
          fv.y += S.y;
        }
        fv.x += v[q].x;
        fv.y += v[q].y;
        cff[o0 + q * ss] = fv;
        r[q].x += uc.x;
        r[q].y += uc.y;
        if (FK == 0 && mean) r[q].x -= k.force;
        r[q].x += k.T5 * fv.x;
        r[q].y += k.T5 * fv.y;
        const double cup = k.aa * RC[j], cdn = k.aa * RC[LP + j];
        r[q].x += cup * (u[q + 2].x - uc.x) - cdn * (uc.x - u[q].x);
        r[q].y += cup * (u[q + 2].y - uc.y) - cdn * (uc.y - u[q].y);
      }
      Sm = S;
    }
  }
  // ---- 2. the forward recurrence from zero; the right-hand side is R on CN
  // rows, the BC value (the (0,0) mode's real part) or zero elsewhere
  double2 g = z2();
  double pa = 1.0;
#pragma unroll
  for (int q = 0; q < K; q++) {
    if (q < nr) {
      const int j = j0 + q;
      const double kind = TB[3 * LP + j], a = TB[j];
      if (kind != (double)ROW_RHS)
        r[q] = make_double2((kind == (double)ROW_BC && mean) ? TB[4 * LP + j] : 0.0, 0.0);
      g.x = r[q].x + a * g.x;
      g.y = r[q].y + a * g.y;
      pa = a * pa;
      r[q] = g;
    }
  }
  // ---- 3. the segment ends carried down the column
  double2 c = carry<MT, +1>(s, m, nseg, make_double2(g.x, g.y), pa, TG, TP);
  // ---- 4. g = local + product x carry, e = g / b; then the backward
  // recurrence x(j) = e(j) + f(j) x(j+1) over the segment (rows >= wlo)
  double pi = 1.0;
#pragma unroll
  for (int q = 0; q < K; q++) {
    if (q < nr) {
      pi = TB[j0 + q] * pi;
      const double rb = TB[LP + j0 + q];
      r[q] = make_double2((r[q].x + pi * c.x) * rb, (r[q].y + pi * c.y) * rb);
    }
  }
  const int qb = wlo > j0 ? wlo - j0 : 0;  // first row of the segment to solve
  double2 xl = z2();
  double ps = 1.0;
#pragma unroll
  for (int q = K - 1; q >= 0; q--) {
    if (q < nr && q >= qb) {
      const double fc = TB[2 * LP + j0 + q];
      xl = make_double2(r[q].x + fc * xl.x, r[q].y + fc * xl.y);
      ps = fc * ps;
      r[q] = xl;
    }
  }
  // ---- 5. the segment starts carried up the column
  c = carry<MT, -1>(s, m, nseg, xl, ps, TG + slots * MT, TP + slots);
  // ---- 6. x = local + product x carry: the post-CN field, rows >= wlo
  double p2 = 1.0;
#pragma unroll
  for (int q = K - 1; q >= 0; q--) {
    if (q < nr && q >= qb) {
      p2 = TB[2 * LP + j0 + q] * p2;
      dst[o0 + q * ss] = make_double2(r[q].x + p2 * c.x, r[q].y + p2 * c.y);
    }
  }
}

// The column stage of field f for modes m0 .. m0+MT-1 of one case.
template <int MT, int K>
__device__ __forceinline__ void col_body(const ColCase &cc, int rk_step, long m0, int f,
                                         const ColLaunch &P, long spin, unsigned extra_tx,
                                         double *sbase) {
  const int NY = cc.C.NY, L = NY + 2, LP = (L + 1) & ~1;  // the case's own row length
  const long ss = cc.C.ss;
  const int mt = (int)((ss - m0) < MT ? (ss - m0) : MT);
  const int wlo = (f >= 3) ? pick(cc.C.JSt, f - 3) - 1 : 1;  // first row solved
  double *TB = sbase;
  double *RC = TB + 5 * P.lp;  // the slots are sized for the largest case
  double2 *TG = reinterpret_cast<double2 *>(RC + 4 * P.lp);
  const int tid = threadIdx.x, npair = blockDim.x / (2 * MT);
  double *TP = reinterpret_cast<double *>(TG + 2 * npair * MT);
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(TP + 2 * npair);
  // the table and grid-factor rows by bulk copies on one mbarrier
  if (tid == 0) dg_mbar_init(bar, 1);
  __syncthreads();
  dg_pdl_wait();  // NL comes from the z-forward kernel
  if (tid == 0) {
    const int nrc = (f == 1) ? 4 : 2;  // grid-factor rows 2..5 (U2) or 0..1
    // extra_tx is 0 except in the wait test, where the barrier then never completes
    dg_mbar_expect_tx(bar, (unsigned)(sizeof(double) * (5 + nrc) * LP) + extra_tx);
    dg_bulk_load(TB, cc.tab + ((long)(rk_step - 1) * (3 + DG_MAX_TH) + f) * 5 * LP,
                 (unsigned)(sizeof(double) * 5 * LP), bar);
    dg_bulk_load(RC, cc.rowc + (long)(f == 1 ? 2 : 0) * LP,
                 (unsigned)(sizeof(double) * nrc * LP), bar);
  }
  const int m = tid % MT, s = tid / MT;
  const int nseg = cc.nseg;
  const bool mine = m < mt && s < nseg;
  const long mg = m < mt ? m0 + m : m0;
  const int j0 = s * K, nr = mine ? min(K, L - j0) : 0;
  const double2 *cu = cc.cu[f], *nl = cc.nl[f], *cpp = cc.cp;
  double2 *cff = cc.cf[f], *dst = cc.out[f];
  int *err = cc.err;
  const FieldCoef k = field_coef(cc, rk_step, f);
  const double KX = cc.kxv[mg % cc.C.nkxp], KZ = cc.kzv[mg / cc.C.nkxp];
  const double k2 = KX * KX + KZ * KZ;
  const double kk = (cc.C.beta == 1.0) ? k2 : pow(k2, cc.C.beta);
  const double Kh = k.T4 * ((f == 2) ? KZ : KX);
  // the table rows have landed (false: they did not within the wait limit)
  auto table = [&]() -> bool {
    const bool landed = dg_mbar_wait(bar, 0, spin);
    if (__syncthreads_or(!landed)) {
      if (tid == 0) {
        atomicExch(err + 1, 1);
        dg_mbar_wait(bar, 0, spin);  // the copies in flight get one more bounded wait
      }
      return false;
    }
    return true;
  };
  const bool old_cf = rk_step > 1;
#define COL_ROWS(FK, CPL)                                                                     \
  col_rows<MT, K, FK, CPL>(k, old_cf, L, ss, mg, j0, nr, nseg, mg == 0, Kh, kk, wlo, cu, nl, cff, \
                        cpp, dst, TB, RC, LP, TG, TP, table)
  if (k.nsrc == 0) {
    if (f == 1) COL_ROWS(1, false);
    else if (f < 3) COL_ROWS(0, false);
    else COL_ROWS(2, false);
  } else {
    if (f == 1) COL_ROWS(1, true);
    else if (f < 3) COL_ROWS(0, true);
    else COL_ROWS(2, true);
  }
#undef COL_ROWS
}

// The column kernel: CTA b takes work[b] = (case, mode tile, field) from
// the case table (every case at substep rk_step with MT modes per CTA).
template <int MT, int K>
__global__ void __launch_bounds__(COL_MAX_THR)
    k_col_cn(const ColCase *__restrict__ cases, const int4 *__restrict__ work, ColLaunch P,
             int rk_step, long spin, unsigned extra_tx) {
  extern __shared__ __align__(16) double cs_raw[];
  const int4 w = work[blockIdx.x];
  col_body<MT, K>(cases[w.x], rk_step, (long)w.y * MT, w.z, P, spin, extra_tx, cs_raw);
}

ColConst make_col_const(const dg_handle *h) {
  ColConst c;
  c.NY = h->NY; c.nf = h->nf; c.nth = h->NTH; c.nkxp = h->nkxp; c.ss = h->ss;
  c.JS = h->jstart; c.JE = h->jend;
  for (int n = 0; n < DG_MAX_TH; n++) {
    c.JSt[n] = h->jstart_th[n]; c.JEt[n] = h->jend_th[n];
    c.ri[n] = h->p.ri[n]; c.pr[n] = h->p.pr[n];
    c.drhodx[n] = h->p.drhodx[n]; c.drhodz[n] = h->p.drhodz[n];
  }
  c.nu = h->p.nu; c.beta = h->p.beta; c.nuv = h->p.nu_v_scale; c.i_ro = h->p.i_ro;
  c.grav_x = h->p.grav_x; c.grav_y = h->p.grav_y; c.grav_z = h->p.grav_z;
  c.px0 = h->p.px0; c.omega0 = h->p.omega0; c.amp_omega0 = h->p.amp_omega0;
  c.f_type = h->p.f_type;
  return c;
}

}  // namespace

// Whether the column stage leaves scalar n in its rhs array (for k_rd_col to
// copy into CU) rather than writing it in place: a velocity right-hand side
// of the same launch reads the scalar's CU when RI * GRAV_x/y/z is nonzero.
bool dg_col_th_to_rhs(const dg_handle *h, int n) {
  const double ri = h->p.ri[n];
  return ri * h->p.grav_x != 0.0 || ri * h->p.grav_y != 0.0 || ri * h->p.grav_z != 0.0;
}

// Per-row grid factors of the column kernel (once per handle, host side).
int dg_col_init(dg_handle *h) {
  const int L = h->NY + 2, LP = (L + 1) / 2 * 2;
  double *t = (double *)calloc((size_t)8 * LP, sizeof(double));
  if (!t) return DG_ERR_OOM;
  const double *dy = h->h_dy, *dyf = h->h_dyf;
  for (int j = 1; j <= h->NY; j++) {
    t[0 * LP + j] = 1.0 / (dy[j + 1] * dyf[j]);
    t[1 * LP + j] = 1.0 / (dy[j] * dyf[j]);
    t[2 * LP + j] = 1.0 / (dyf[j] * dy[j]);
    t[3 * LP + j] = 1.0 / (dyf[j - 1] * dy[j]);
    t[6 * LP + j] = 1.0 / dyf[j];
    t[7 * LP + j] = (j >= 2 && j < h->NY) ? 1.0 / (dy[j + 1] * dyf[j]) : 0.0;
  }
  for (int j = 1; j < L; j++) t[4 * LP + j] = 1.0 / dy[j];
  for (int j = 0; j < L; j++) t[5 * LP + j] = dyf[j];
  cudaError_t e = dg_malloc(h, (void **)&h->rowc, sizeof(double) * 8 * LP);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->rowc, t, sizeof(double) * 8 * LP, cudaMemcpyHostToDevice, h->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
  free(t);
  DG_CUDA(e);
  return DG_OK;
}

static int col_segk(const dg_handle *h) { return h->NY + 2 <= SEG_SHORT ? SEG_KS : SEG_K; }
static int col_nseg(const dg_handle *h) { return dg_cdiv(h->NY + 2, col_segk(h)); }

// threads of one CTA for handle h at mt modes: one per (mode, segment)
static int col_threads(const dg_handle *h, int mt) {
  return (mt * col_nseg(h) + 31) / 32 * 32;
}

// launch sizes of handle h alone (nwork left 0)
static ColLaunch col_sizes(const dg_handle *h) {
  ColLaunch P;
  P.lp = (h->NY + 2 + 1) / 2 * 2;
  P.nwork = 0;
  return P;
}

size_t dg_col_smem(const dg_handle *h, int mt) {
  return col_smem_l(col_sizes(h), mt, col_threads(h, mt));
}

// the case description of handle h
static void fill_case(dg_handle *h, ColCase *cc) {
  memset(cc, 0, sizeof(*cc));
  cc->C = make_col_const(h);
  cc->dscal = h->dscal;
  cc->tab = h->cn_tab;
  cc->kxv = h->kx;
  cc->kzv = h->kz;
  cc->rowc = h->rowc;
  for (int f = 0; f < h->nf; f++) {
    cc->cu[f] = h->cu[f];
    cc->nl[f] = h->rhs[f];
    cc->cf[f] = h->cf[f];
    cc->out[f] = (f < 3 || dg_col_th_to_rhs(h, f - 3)) ? h->rhs[f] : h->cu[f];
  }
  cc->cp = h->cp;
  cc->err = h->dflag;
  cc->nseg = col_nseg(h);
}

// modes per CTA for handle h: the tuned value, halved until the CTA fits
// (one thread per mode and segment)
static int col_mt(const dg_handle *h, int want) {
  int mt = want;
  while (mt > 2 && (dg_col_smem(h, mt) > 220 * 1024 || col_threads(h, mt) > COL_MAX_THR)) mt /= 2;
  return mt;
}

static int col_fits(const dg_handle *h, int mt) {
  if (dg_col_smem(h, mt) > 220 * 1024 || col_threads(h, mt) > COL_MAX_THR) {
    char b[96];
    snprintf(b, sizeof(b), "column kernel: NY too large for two modes per CTA (NY + 2 <= %d)",
             COL_MAX_THR / 2 * SEG_K);
    dg_set_error(b);
    return DG_ERR_DIMS;
  }
  return DG_OK;
}

int dg_col_mt_eff(const dg_handle *h) { return col_mt(h, h->cn_mt); }

int dg_col_class(const dg_handle *h) { return dg_col_mt_eff(h) * 64 + col_segk(h); }

// the work list of one case: (case c, tile, field, 0) per item
static void case_work(const dg_handle *h, int c, int mt, std::vector<int4> &work) {
  const int tiles = dg_cdiv(h->ss, mt);
  for (int f = 0; f < h->nf; f++)
    for (int t = 0; t < tiles; t++) work.push_back(make_int4(c, t, f, 0));
}

// The handle's device copy of its one-case table and work list for mt,
// rebuilt when mt changes.  The copies are synchronous, so they cannot run
// inside a stream capture: diablo_step's first step of a kind, which runs
// eagerly, builds them before any capture.
static int col_tables(dg_handle *h, int mt) {
  if (h->col_dcase && h->col_dmt == mt) return DG_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
    dg_set_error("the column kernel's case table must be built before a stream capture "
                 "(run one substep eagerly after changing the tuning)");
    return DG_ERR_ARG;
  }
  ColCase cc;
  fill_case(h, &cc);
  std::vector<int4> work;
  case_work(h, 0, mt, work);
  DG_CUDA(cudaStreamSynchronize(h->st));
  if (h->col_dcase) dg_free(h, h->col_dcase);
  if (h->col_dwork) dg_free(h, h->col_dwork);
  h->col_dcase = nullptr;
  h->col_dwork = nullptr;
  DG_CUDA(dg_malloc(h, &h->col_dcase, sizeof(cc)));
  DG_CUDA(dg_malloc(h, (void **)&h->col_dwork, sizeof(int4) * work.size()));
  DG_CUDA(cudaMemcpyAsync(h->col_dcase, &cc, sizeof(cc), cudaMemcpyHostToDevice, h->st));
  DG_CUDA(cudaMemcpyAsync(h->col_dwork, work.data(), sizeof(int4) * work.size(),
                          cudaMemcpyHostToDevice, h->st));
  DG_CUDA(cudaStreamSynchronize(h->st));
  h->col_dmt = mt;
  h->col_dnwork = (int)work.size();
  return DG_OK;
}

static int launch_col(cudaStream_t st, int pdl, const dg_col_launch &cl, const void *dev_cases,
                      const int4 *dev_work, int rk_step, long spin, unsigned extra_tx) {
  ColLaunch P;
  P.lp = cl.lp;
  P.nwork = cl.nwork;
#define CS_CASE(MTV, KV)                                                                        \
  if (cl.mt == MTV && cl.segk == KV) {                                                          \
    dg_big_smem((const void *)k_col_cn<MTV, KV>);                                               \
    DG_CUDA(dg_launch(pdl, k_col_cn<MTV, KV>, dim3(cl.grid), dim3(cl.thr), cl.smem, st,         \
                      (const ColCase *)dev_cases, dev_work, P, rk_step, spin, extra_tx));       \
  }
  CS_CASE(2, SEG_K) CS_CASE(4, SEG_K) CS_CASE(8, SEG_K) CS_CASE(16, SEG_K)
  CS_CASE(2, SEG_KS) CS_CASE(4, SEG_KS) CS_CASE(8, SEG_KS) CS_CASE(16, SEG_KS)
#undef CS_CASE
  DG_LAUNCHED();
  return DG_OK;
}

// launch sizes of handles hs together at `want` modes per CTA: the largest
// any of them needs (a case's CTAs leave threads beyond its own segments idle)
static int col_plan(dg_handle *const *hs, int n, int want, int nwork, dg_col_launch *cl) {
  int mt = want;
  for (int c = 0; c < n; c++) mt = std::min(mt, col_mt(hs[c], want));
  dg_col_launch r = {};
  r.mt = mt;
  r.segk = col_segk(hs[0]);
  for (int c = 0; c < n; c++) {
    if (col_segk(hs[c]) != r.segk) {
      dg_set_error("column kernel: columns with different segments cannot share a launch");
      return DG_ERR_ARG;
    }
    DG_TRY(col_fits(hs[c], mt));
    r.lp = std::max(r.lp, col_sizes(hs[c]).lp);
    r.thr = std::max(r.thr, col_threads(hs[c], mt));
  }
  ColLaunch P;
  P.lp = r.lp;
  P.nwork = nwork;
  r.smem = col_smem_l(P, mt, r.thr);
  if (r.smem > 220 * 1024) {
    dg_set_error("column kernel: the cases' tables do not fit in shared memory");
    return DG_ERR_DIMS;
  }
  r.nwork = nwork;
  r.grid = nwork;  // one CTA per work item
  *cl = r;
  return DG_OK;
}

// The column stage of substep rk_step: right-hand sides and CN solves of
// every field (k_col_cn; the post-CN fields land in the rhs arrays), then,
// when rd, REM_DIV and the pressure update from there into CU (k_rd_col).
// rd = false leaves REM_DIV to the caller (COURANT runs between them).
int dg_col_step_dev(dg_handle *h, int rk_step, bool rd) {
  if (h->tables_pending) {
    DG_CUDA(cudaStreamWaitEvent(h->st, h->ev_join, 0));
    h->tables_pending = false;
  }
  const int mt = col_mt(h, h->cn_mt);
  DG_TRY(col_fits(h, mt));
  DG_TRY(col_tables(h, mt));
  dg_col_launch cl;
  dg_handle *hs[1] = {h};
  DG_TRY(col_plan(hs, 1, mt, h->col_dnwork, &cl));
  // the wait test (DG_TUNE_WAIT_TEST) applies to this one launch
  const long spin = h->wait_test > 0 ? (long)h->wait_test : DG_ASYNC_SPIN;
  const unsigned extra_tx = h->wait_test > 0 ? 16u : 0u;
  h->wait_test = 0;
  dg_kt_begin(h, "k_col_cn", h->st);
  DG_TRY(launch_col(h->st, h->pdl, cl, h->col_dcase, h->col_dwork, rk_step, spin, extra_tx));
  if (rd) DG_TRY(dg_rem_div_dev(h, 1, rk_step, true));
  return DG_OK;
}

// ---------------------------------------------------------- ragged launch
// The column stage of several cases at the same substep in one launch (the
// ensemble server's groups).  dg_col_batch_build fills, for the handles, the
// host images of the case table and the work list (one (case, tile, field)
// entry per item) with one MT for all, and the launch sizes; the caller
// copies the images to device memory it owns and launches with
// dg_col_batch_launch.  Each case's REM_DIV follows on its own stream.
// Results do not depend on the batch: each mode's arithmetic is the
// single-case launch's, with the same kernel.
int dg_col_batch_build(dg_handle *const *hs, int n, int want_mt, std::vector<unsigned char> &cases,
                       std::vector<int4> &work, dg_col_launch *cl) {
  int mt = want_mt;
  for (int c = 0; c < n; c++) mt = std::min(mt, col_mt(hs[c], want_mt));
  cases.assign(sizeof(ColCase) * n, 0);
  work.clear();
  for (int c = 0; c < n; c++) {
    ColCase cc;
    fill_case(hs[c], &cc);
    memcpy(cases.data() + sizeof(ColCase) * c, &cc, sizeof(ColCase));
    case_work(hs[c], c, mt, work);
  }
  return col_plan(hs, n, mt, (int)work.size(), cl);
}

int dg_col_batch_launch(cudaStream_t st, const dg_col_launch &cl, const void *dev_cases,
                        const int4 *dev_work, int rk_step) {
  return launch_col(st, 0, cl, dev_cases, dev_work, rk_step, DG_ASYNC_SPIN, 0u);
}
