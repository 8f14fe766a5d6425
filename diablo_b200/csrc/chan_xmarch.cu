// The x-row stage of a channel substep for rows of 256 (with scalars), 384 and
// 512 points, in FP32 of 192 and 256 too, which have too many points for the
// registers of k_xrows (chan_xrows.cuh): x c2r of every field, the products of
// for/channel.f:409-571,665-720 and their x r2c, one CTA per z-row marching
// up through a chunk of planes.
//
// A row of NX = R1 T points is one point column per thread: thread t holds
// x = t + T r, r = 0..R1-1, of the planes j and j+1 in registers (plane j-1
// in its own shared-memory slots).  That makes one radix-R1 pass of every
// transform a register operation, and leaves R1 independent transforms of
// length T per signal, which warps run in place without a CTA barrier:
//   inverse, k = R1 m + q:  y_q(b) = sum_m X(R1 m + q) W_T^(-b m)   (warps)
//            x(t + T r) = sum_q W_R1^(-r q) (W_N^(-t q) y_q(t))     (threads)
//   forward: y_q(t) = W_N^(t q) sum_r x(t + T r) W_R1^(r q)         (threads)
//            X(R1 m + q) = sum_b y_q(b) W_T^(b m)                   (warps)
// The first pass of the inverse takes its inputs from global memory (two
// fields' spectra packed into one complex signal) and the radix-R1 passes
// work on registers, so a row makes 4 trips through shared memory on the way
// to points and 5.7 on the way back, for 8 each with a buffer between every
// pass; the physical rows never reach HBM.  What bounds it is shared-memory
// bandwidth: about 350 KB of it per row and plane at NX = 512 with a scalar.
//
// At 512x257x384 with a scalar it takes 2.12 ms per launch in FP64 (1.43 in
// FP32), where a c2r launch into an array of physical rows and a launch per
// product pair took 1.20 + 3.39 ms (0.60 + 3.63); 0.21 ms at 192x193x192 in FP32
// (0.06 + 0.38).  ncu at 512x65x384: shared memory busy 47% of the time, 12
// warps per SM (168 registers), waiting mostly on HBM and shared memory; the row
// that the next step reads is prefetched into L2 (653 -> 620 us there).  Sub-
// transforms that start with radix 8 (more registers for twiddles in the radix-16
// pass after it) measured slower: 753 us.
//
// The products are the pairs of k_xprod (chan_kernels.cu): the flux
// differences are taken in physical space, so each pair maps onto the A/B
// arrays of G.  With FP32 (mixed precision) every row is split into its mean
// (FP64) and its fluctuation, and the means of the products are summed in
// FP64 and put in the kx = 0 bin.
#include <math.h>

#include <type_traits>

#include "dg_internal.cuh"
#include "fft.cuh"

using namespace dgfft;

namespace {

// stride of a sub-transform's buffer: at least the padded length, and such
// that the lanes of a quarter warp (half warp for 8-byte values), which read
// consecutive bins k = R1 m + q, fall into different banks
__host__ __device__ constexpr int xm_sstr(int T, int R1, int esz) {
  const int w = esz == 16 ? 8 : 16;
  // (8-byte values: a half warp of the passes with T/R = 8 covers two
  // sub-transforms, whose buffers then must lie 8 values apart)
  const int want = esz == 16 ? (R1 == 3 ? 3 : 2) : 8;  // R1 is 3 or 4
  int s = T + (T - 1) / 16;
  while (s % w != want) s++;
  return s;
}

__host__ __device__ constexpr int xm_pairs(int nth) { return 4 + nth + (nth + 1) / 2; }
__host__ __device__ constexpr int xm_signals(int nth) {
  return xm_pairs(nth) > (4 + nth) / 2 ? xm_pairs(nth) : (4 + nth) / 2;
}

// fields of the inverse's signal s: (U1, TH1), TH1 scaled to U1's magnitude
// (dg_pair_shift); (U2, U3), (TH2, -)
__host__ __device__ constexpr int xm_fa(int s) { return s < 2 ? s : 2 * s; }
__host__ __device__ constexpr int xm_fb(int s) { return s == 0 ? 3 : s == 1 ? 2 : 2 * s + 1; }

struct XmArgs {
  int NY, NZ;
  long Hfield, Gfield;
  int chunk, jbase, jtop;
  const double *dyf, *dy, *kx;
  const unsigned *peak;  // of H's planes
  int planes, plen;
};

// first pass of the inverse sub-transforms s0 .. s0+ns-1: radix R, inputs
// from load(sub, m), no twiddles
template <int T, int R, typename CX, typename Load>
__device__ __forceinline__ void xm_first(CX *__restrict__ buf, int s0, int ns, int sstr, int lane,
                                         Load load) {
  constexpr int NB = T / R;
  static_assert(NB <= 32, "warp pass needs T/R <= 32");
  constexpr int SPR = 32 / NB;
  const int sl = lane / NB, b = lane % NB;
  for (int a = 0; a < ns; a += SPR) {
    const int s = a + sl;
    if (sl < SPR && s < ns) {
      CX v[R];
      load(s0 + s, b, v);
      dft<R>(v, +1);
      CX *out = buf + (s0 + s) * sstr;
#pragma unroll
      for (int r = 0; r < R; r++) out[pad(b * R + r)] = v[r];
    }
  }
  __syncwarp();
}

// hides a value's origin from the compiler, so that what is computed from it
// inside the plane loop is not kept in registers across it (FP64, T = 64:
// 4% faster per launch; the others measured slower with it)
template <bool ON>
__device__ __forceinline__ int xm_fresh(int v) {
  if constexpr (ON) asm volatile("" : "+r"(v));
  return v;
}

// passes P.. of the sub-transforms; the last one leaves out the rows of its
// outputs that lie wholly in (LO, HI)
template <int T, int SIGN, int P, int LO, int HI, typename CX>
__device__ __forceinline__ void xm_passes(CX *__restrict__ buf, int nsig, int sstr,
                                          const CX *__restrict__ tw, int lane) {
  constexpr int R = plan_radix(T, P), NS = plan_ns(T, P), NB = T / R;
  constexpr bool LAST = P + 1 == plan_passes(T);
  const CX *twp = tw + twp_off<T, 0>(P);
  if constexpr (!LAST || LO >= HI) {
    wpass<T, R, NS, SIGN, true>(buf, nsig, sstr, twp, lane);
  } else {
    static_assert(NS == NB, "the last pass spans the transform");
    constexpr int SPR = 32 / NB;
    const int sl = lane / NB, b = lane % NB;
    for (int s0 = 0; s0 < nsig; s0 += SPR) {
      const int s = s0 + sl;
      const bool act = (sl < SPR) && (s < nsig);
      CX v[R];
      if (act) {
        const CX *in = buf + s * sstr;
#pragma unroll
        for (int r = 0; r < R; r++) {
          CX x = in[pad(b + r * NB)];
          if (P > 0 && r > 0) {
            CX t = twp[r * NS + b];
            if (SIGN > 0) t.y = -t.y;
            x = cmul(x, t);
          }
          v[r] = x;
        }
        dft<R>(v, SIGN);
      }
      __syncwarp();
      if (act) {
        CX *out = buf + s * sstr;
#pragma unroll
        for (int r = 0; r < R; r++)
          if (!(r * NB > LO && r * NB + NB - 1 < HI)) out[pad(b + r * NB)] = v[r];
      }
      __syncwarp();
    }
  }
  if constexpr (!LAST) xm_passes<T, SIGN, P + 1, LO, HI>(buf, nsig, sstr, tw, xm_fresh<T == 64 && sizeof(CX) == 16>(lane));
}

// the sum over the lanes of each of the first NM of 16 values: lane l ends
// with the total of value (l >> 1) (halving the values kept with every step)
template <int NM>
__device__ __forceinline__ double xm_lane_sums(double (&v)[16], int lane) {
#pragma unroll
  for (int i = NM; i < 16; i++) v[i] = 0.0;
#pragma unroll
  for (int o = 16, n = 8; o >= 2; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const double keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// out of line: inlined, it moved the register allocation of the plane loop (512 points
// with a scalar in FP64: 588 bytes of spills and 2.82 ms per launch, 232 and 2.12 so)
template <typename T, int NTH>
__device__ __noinline__ void xm_plane_shifts(int *sh, const unsigned *peak, int planes, int len,
                                             int pl0, int n) {
  dg_plane_shifts<T, NTH>(sh, peak, planes, len, pl0, n);
}

template <int T, int R1, int NTH, typename CX>
__global__ void __launch_bounds__(T, (T == 128 ? 1 : 2) * (sizeof(CX) == 16 ? 3 : 4)) k_xmarch(
    XmArgs A, const CX *__restrict__ H, const CX *__restrict__ tw, CX *__restrict__ G) {
  using TR = typename CT<CX>::T;
  constexpr bool F32 = sizeof(TR) == 4;
  constexpr int NX = T * R1, NKXP = NX / 3 + 1;
  constexpr int NF = 3 + NTH, NPIN = (NF + 1) / 2, NPP = xm_pairs(NTH), NM = 8 + 3 * NTH;
  constexpr int SSTR = xm_sstr(T, R1, (int)sizeof(CX));
  constexpr int NW = T / 32;
  static_assert(tp_ok(T), "the sub-transforms read per-pass tables");
  // bins NX/3 + 1 .. NX - NX/3 - 1 are zero on the way to points and not
  // wanted on the way back
  constexpr int KLO = NX / 3, KHI = NX - NX / 3;
  extern __shared__ double2 sm_raw[];
  CX *stw = reinterpret_cast<CX *>(sm_raw);       // twiddles of length T
  CX *buf = stw + T;                              // [signal][q][SSTR]
  TR *prv = reinterpret_cast<TR *>(buf + xm_signals(NTH) * R1 * SSTR);  // [field][r][T], plane j-1
  int *shf = reinterpret_cast<int *>(prv + NF * NX);  // shifts of the chunk's planes
  __shared__ double red[F32 ? NW : 1][16];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int z = blockIdx.x, NZ = A.NZ;
  // W_T^m = W_N^(R1 m)
  for (int i = t; i < twp_len<T, 0>(); i += T) {
    int p = 1;
    while (i >= twp_off<T, 0>(p + 1)) p++;
    const int R = plan_radix(T, p), NS = plan_ns(T, p);
    const int e = i - twp_off<T, 0>(p), r = e / NS, k = e - r * NS;
    stw[i] = tw[r * k * (T / (NS * R)) * R1];
  }
  CX w[R1];
#pragma unroll
  for (int q = 1; q < R1; q++) w[q] = tw[t * q];
  dg_pdl_wait();  // H comes from the z inverse
  __syncthreads();
  const int j0 = A.jbase + blockIdx.y * A.chunk;
  const int j1 = min(j0 + A.chunk - 1, A.jtop);
  const long plane = (long)NZ * NKXP;
  const CX *Hz = H + (long)z * NKXP;

  TR cur[NF][R1], nxt[NF][R1];
  double dcur[NF], dnxt[NF], dprv[NF];  // row means (FP32 form)

  if constexpr (NTH > 0)
    xm_plane_shifts<TR, NTH>(shf, A.peak, A.planes, A.plen, j0 - 1, j1 - j0 + 3);
  int shc = 0, shn = 0;  // two scalars: TH2's shift to TH1 in their common pair, planes j and j+1
  auto load_plane = [&](int pl, TR (&dst)[NF][R1], double (&dcv)[NF], int &sh) {
    const CX *row = Hz + (long)pl * plane;
    const int sw = NTH > 0 ? shf[pl - j0 + 1] : 0, d = (short)sw;  // TH1 goes times 2^d
    if constexpr (F32) {
#pragma unroll
      for (int f = 0; f < NF; f++) dcv[f] = (double)__ldg(row + f * A.Hfield).x;
    }
    if constexpr (NTH == 2) {
      if constexpr (F32)  // the products hold the row means, the peaks do not
        sh = dg_pair_shift<TR>(max((sw >> 24) & 255, dg_mag_exp<TR>(dg_mag((TR)dcv[3]))),
                               max((sw >> 16) & 255, dg_mag_exp<TR>(dg_mag((TR)dcv[4]))), 0);
      else
        sh = sw >> 16;
    }
    constexpr int NS = NPIN * R1, PER = (NS + NW - 1) / NW;
    const int ln = xm_fresh<T == 64 && sizeof(CX) == 16>(lane), s0 = xm_fresh<T == 64 && sizeof(CX) == 16>(warp) * PER, ns = min(PER, NS - s0);
    if (ns > 0) {
      constexpr int R0 = plan_radix(T, 0), NB0 = T / R0;
      xm_first<T, R0>(buf, s0, ns, SSTR, ln, [&](int sub, int b, CX *v) {
        const int q = sub % R1, s = sub / R1, fb = xm_fb(s);
        const CX *ra = row + xm_fa(s) * A.Hfield, *rb = row + fb * A.Hfield;
        const bool two = fb < NF;
        const TR sc = dg_pow2<TR>(NTH > 0 && s == 0 ? d : 0);
#pragma unroll
        for (int r = 0; r < R0; r++) {
          if (R1 * r * NB0 > KLO && R1 * (r * NB0 + NB0) - 1 < KHI) {
            v[r] = CT<CX>::mk(0, 0);
            continue;
          }
          const int k = R1 * (b + r * NB0) + q;
          const int kk = (k <= NX / 2) ? k : NX - k;
          CX a = CT<CX>::mk(0, 0), c = CT<CX>::mk(0, 0);
          if (kk < NKXP && !(F32 && kk == 0)) {
            a = __ldg(ra + kk);
            if (two) c = __ldg(rb + kk);
            if (kk == 0) a.y = c.y = 0;
          }
          v[r] = (k == kk) ? CT<CX>::mk(a.x - sc * c.y, a.y + sc * c.x)
                           : CT<CX>::mk(a.x + sc * c.y, sc * c.x - a.y);
        }
      });
      xm_passes<T, +1, 1, 0, 0>(buf + s0 * SSTR, ns, SSTR, stw, xm_fresh<T == 64 && sizeof(CX) == 16>(ln));
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NPIN; s++) {
      CX v[R1];
#pragma unroll
      for (int q = 0; q < R1; q++) {
        v[q] = buf[(s * R1 + q) * SSTR + pad(t)];
        if (q > 0) v[q] = cmul(v[q], conjg(w[q]));
      }
      dft<R1>(v, +1);
#pragma unroll
      for (int r = 0; r < R1; r++) {
        dst[xm_fa(s)][r] = v[r].x;
        if (xm_fb(s) < NF)
          dst[xm_fb(s)][r] = s == 0 ? v[r].y * dg_pow2<TR>(-d) : v[r].y;
      }
    }
    __syncthreads();
  };

  load_plane(j0 - 1, cur, dprv, shc);
#pragma unroll
  for (int f = 0; f < NF; f++)
#pragma unroll
    for (int r = 0; r < R1; r++) prv[(f * R1 + r) * T + t] = cur[f][r];
  load_plane(j0, cur, dcur, shc);
  for (int j = j0; j <= j1; j++) {
    // the row that the next step reads comes from HBM: into L2 meanwhile
    if (j < j1) {
      constexpr int LINES = (NKXP * (int)sizeof(CX) + 127) / 128;
      for (int i = t; i < NF * LINES; i += T) {
        const char *row = reinterpret_cast<const char *>(Hz + (i / LINES) * A.Hfield + (j + 2) * plane);
        const int off = min((i % LINES) * 128, NKXP * (int)sizeof(CX) - 1);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + off));
      }
    }
    load_plane(j + 1, nxt, dnxt, shn);
    const double dyfj = A.dyf[j], dyfm = A.dyf[j - 1], wgyd = 1.0 / (2.0 * A.dy[j]);
    const TR cj = (TR)(dyfj * wgyd), cm = (TR)(dyfm * wgyd);
    double acc[16];  // FP32 form: sums of the products of the fluctuations
    if constexpr (F32) {
#pragma unroll
      for (int i = 0; i < NM; i++) acc[i] = 0.0;
    }
    // the pairs at the thread's points, one signal at a time: the radix-R1
    // pass in registers, then y_q to shared memory
    auto old = [&](int f, int r) -> TR { return prv[(f * R1 + r) * T + t]; };
    // FP32 form: (D1 + a)(D2 + b) without its mean part D1 D2; the sum of a b
    // goes to accumulator m in FP64
    auto pr = [&](double d1, TR a, double d2, TR b, int m, double sg) -> TR {
      if constexpr (F32) acc[m] = fma(sg * (double)a, (double)b, acc[m]);
      return (TR)sg * ((TR)d1 * b + (TR)d2 * a + a * b);
    };
    // (X(j+1) + X(j)) U2(j+1) - (X(j) + X(j-1)) U2(j)
    auto rise = [&](int f, int r, int m) -> TR {
      const TR x = cur[f][r], xp = nxt[f][r] + x, xm = x + old(f, r);
      if constexpr (F32)
        return pr(dnxt[f] + dcur[f], xp, dnxt[1], nxt[1][r], m, 1.0) +
               pr(dcur[f] + dprv[f], xm, dcur[1], cur[1][r], m, -1.0);
      else
        return xp * nxt[1][r] - xm * cur[1][r];
    };
    // F(f) F(g) at plane j
    auto prod = [&](int f, int g, int r, int m) -> TR {
      if constexpr (F32) return pr(dcur[f], cur[f][r], dcur[g], cur[g][r], m, 1.0);
      else return cur[f][r] * cur[g][r];
    };
    // Ubar U2 at GY j
    auto ubar = [&](int f, int r, int m) -> TR {
      const TR x = cj * cur[f][r] + cm * old(f, r);
      if constexpr (F32)
        return pr((dyfj * dcur[f] + dyfm * dprv[f]) * wgyd, x, dcur[1], cur[1][r], m, 1.0);
      else
        return x * cur[1][r];
    };
    auto pair_at = [&](int s, int r) -> CX {
      if (s == 0) return CT<CX>::mk(prod(2, 0, r, 0), rise(2, r, 1));
      if (s == 1) return CT<CX>::mk(prod(0, 0, r, 2), rise(0, r, 3));
      if (s == 2) {
        const TR gp = (TR)0.5 * (cur[1][r] + nxt[1][r]), gm = (TR)0.5 * (old(1, r) + cur[1][r]);
        TR b;
        if constexpr (F32) {
          const double gpd = 0.5 * (dcur[1] + dnxt[1]), gmd = 0.5 * (dprv[1] + dcur[1]);
          b = pr(gpd, gp, gpd, gp, 5, 1.0) + pr(gmd, gm, gmd, gm, 5, -1.0);
        } else {
          b = gp * gp - gm * gm;
        }
        return CT<CX>::mk(ubar(0, r, 4), b);
      }
      if (s == 3) return CT<CX>::mk(ubar(2, r, 6), prod(2, 2, r, 7));
      if (s < 4 + NTH) {
        const int f = s - 1, m = 2 * s;
        return CT<CX>::mk(prod(f, 0, r, m), rise(f, r, m + 1));
      }
      const int n = 2 * (s - 4 - NTH), m = 8 + 2 * NTH + n;
      return CT<CX>::mk(
          prod(3 + n, 2, r, m),
          n + 1 < NTH ? dg_pow2<TR>(shc) * prod(4 + n < NF ? 4 + n : 3, 2, r, m + 1) : (TR)0);
    };
#pragma unroll
    for (int s = 0; s < NPP; s++) {
      CX P[R1];
#pragma unroll
      for (int r = 0; r < R1; r++) P[r] = pair_at(s, r);
      dft<R1>(P, -1);
#pragma unroll
      for (int q = 0; q < R1; q++)
        buf[(s * R1 + q) * SSTR + pad(t)] = q > 0 ? cmul(P[q], w[q]) : P[q];
    }
    if constexpr (F32) {
      const double v = xm_lane_sums<NM>(acc, lane);
      if ((lane & 1) == 0) red[warp][lane >> 1] = v;
    }
    // plane j becomes j-1, j+1 becomes j
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
      for (int r = 0; r < R1; r++) {
        prv[(f * R1 + r) * T + t] = cur[f][r];
        cur[f][r] = nxt[f][r];
      }
    __syncthreads();
    {
      constexpr int NS = NPP * R1, PER = (NS + NW - 1) / NW;
      const int s0 = xm_fresh<T == 64 && sizeof(CX) == 16>(warp) * PER, ns = min(PER, NS - s0);
      if (ns > 0)
        xm_passes<T, -1, 0, KLO / R1, KHI / R1>(buf + s0 * SSTR, ns, SSTR, stw, xm_fresh<T == 64 && sizeof(CX) == 16>(lane));
    }
    __syncthreads();
    const double id2 = 1.0 / (2.0 * dyfj), idyj = 1.0 / A.dy[j];
    constexpr double hx = 0.5 / (double)NX;
#pragma unroll 1
    for (int k = xm_fresh<T == 64 && sizeof(CX) == 16>(t); k < NKXP; k += T) {
      const int km = (NX - k) % NX;
      const CX *bk = buf + (k % R1) * SSTR + pad(k / R1);
      const CX *bm = buf + (km % R1) * SSTR + pad(km / R1);
      const double KX = A.kx[k];
      CX *o = G + (long)j * plane + (long)z * NKXP + k;
#pragma unroll
      for (int s = 0; s < NPP; s++) {
        const CX zk = bk[s * R1 * SSTR], zm = bm[s * R1 * SSTR];
        // the pair's members, scaled by 1/NX: A = (Z_k + conj Z_{N-k})/2,
        // B = -i/2 (Z_k - conj Z_{N-k})
        double2 a = make_double2(hx * ((double)zk.x + zm.x), hx * ((double)zk.y - zm.y));
        double2 b = make_double2(hx * ((double)zk.y + zm.y), -hx * ((double)zk.x - zm.x));
        if (NTH == 2 && s == 4 + NTH) {
          b.x *= dg_pow2<double>(-shc);
          b.y *= dg_pow2<double>(-shc);
        }
        if constexpr (F32) {
          if (k == 0) {
            // the row means of the pair's products
            const double *c = dcur, *n = dnxt, *p = dprv;
            int ma = 2 * s, mb = 2 * s + 1;
            double da, db = 0.0;
            if (s == 0) {
              da = c[2] * c[0];
              db = (n[2] + c[2]) * n[1] - (c[2] + p[2]) * c[1];
            } else if (s == 1) {
              da = c[0] * c[0];
              db = (n[0] + c[0]) * n[1] - (c[0] + p[0]) * c[1];
            } else if (s == 2) {
              const double gpd = 0.5 * (c[1] + n[1]), gmd = 0.5 * (p[1] + c[1]);
              da = (dyfj * c[0] + dyfm * p[0]) * wgyd * c[1];
              db = gpd * gpd - gmd * gmd;
            } else if (s == 3) {
              da = (dyfj * c[2] + dyfm * p[2]) * wgyd * c[1];
              db = c[2] * c[2];
            } else if (s < 4 + NTH) {
              const int i = s - 4;
              da = c[3 + i] * c[0];
              db = (n[3 + i] + c[3 + i]) * n[1] - (c[3 + i] + p[3 + i]) * c[1];
            } else {
              const int i = 2 * (s - 4 - NTH);
              ma = 8 + 2 * NTH + i;
              mb = ma + 1;
              da = c[3 + i] * c[2];
              if (i + 1 < NTH) db = c[4 + i < NF ? 4 + i : 3] * c[2];
            }
            double sa = 0.0, sb = 0.0;
#pragma unroll
            for (int x = 0; x < NW; x++) {
              sa += red[x][ma];
              if (mb < NM) sb += red[x][mb];
            }
            a = make_double2(da + sa / (double)NX, 0.0);
            b = make_double2(db + sb / (double)NX, 0.0);
          }
        }
        // -i kx A - c B
        auto flux = [&](double c) {
          return CT<CX>::mk((TR)(KX * a.y - b.x * c), (TR)(-KX * a.x - b.y * c));
        };
        const CX ac = CT<CX>::mk((TR)a.x, (TR)a.y), bc = CT<CX>::mk((TR)b.x, (TR)b.y);
        if (s == 0) {
          o[0] = ac;                     // U1: A = U1U3
          o[5 * A.Gfield] = flux(id2);   // U3: B = -ikx U1U3 - (fl3(j+1) - fl3(j)) / (2 DYF)
        } else if (s == 1) {
          o[A.Gfield] = flux(id2);       // U1: B = -ikx U1U1 - (fl1(j+1) - fl1(j)) / (2 DYF)
        } else if (s == 2) {
          o[3 * A.Gfield] = flux(idyj);  // U2: B = -ikx Ubar1 U2 - (g(j) - g(j-1)) / DY
        } else if (s == 3) {
          o[2 * A.Gfield] = ac;          // U2: A = Ubar3 U2
          o[4 * A.Gfield] = bc;          // U3: A = U3U3
        } else if (s < 4 + NTH) {
          o[(7 + 2 * (s - 4)) * A.Gfield] = flux(id2);  // TH: B = -ikx TH U1 - dflth / (2 DYF)
        } else {
          const int i = 2 * (s - 4 - NTH);
          o[(6 + 2 * i) * A.Gfield] = ac;               // TH: A = TH U3
          if (i + 1 < NTH) o[(8 + 2 * i) * A.Gfield] = bc;
        }
      }
    }
    shc = shn;
    if constexpr (F32) {
#pragma unroll
      for (int f = 0; f < NF; f++) {
        dprv[f] = dcur[f];
        dcur[f] = dnxt[f];
      }
    }
    __syncthreads();  // the next plane's transforms reuse the buffers
  }
}

// three CTAs of 128 threads per SM in FP64 (168 registers; 71 KB of shared
// memory at NX = 512 with a scalar), four in FP32 (128 registers: 485 -> 390 us
// at 512x65x384 with a scalar)
template <int T, int R1, int NTH, typename CX>
size_t xm_smem(int ny) {
  return sizeof(CX) * (T + (size_t)xm_signals(NTH) * R1 * xm_sstr(T, R1, (int)sizeof(CX))) +
         sizeof(typename CT<CX>::T) * (3 + NTH) * (size_t)T * R1 + (NTH > 0 ? sizeof(int) * (ny + 2) : 0);
}

template <int T, int R1, int NTH, typename CX>
int xm_launch(dg_handle *h, const CX *H, const CX *tw, CX *G, const char *name) {
  auto kern = k_xmarch<T, R1, NTH, CX>;
  const size_t sm = xm_smem<T, R1, NTH, CX>(h->NY);
  dg_big_smem((const void *)kern);
  XmArgs A;
  A.NY = h->NY; A.NZ = h->NZ;
  A.Hfield = A.Gfield = (long)h->nplanes * h->NZ * h->nkxp;
  A.jbase = 1; A.jtop = h->NY;
  A.dyf = h->dyf; A.dy = h->dy; A.kx = h->kx;
  A.peak = h->peak; A.planes = h->NY + 2; A.plen = h->peak_len;
  A.chunk = h->xrow_chunk > 0 ? (h->xrow_chunk < h->NY ? h->xrow_chunk : h->NY)
                              : dg_march_chunk(h->NY, h->NZ, (const void *)kern, T, sm, 1.0, 0.7);
  dg_kt_begin(h, name, h->st);
  DG_CUDA(dg_launch(h->pdl, kern, dim3(h->NZ, dg_cdiv(h->NY, A.chunk)), dim3(T), sm, h->st, A, H, tw,
                    G));
  DG_LAUNCHED();
  return DG_OK;
}

template <typename CX>
int xm_dispatch(dg_handle *h, const CX *H, const CX *tw, CX *G, const char *name) {
#define XM_CASE(T, R1)                                               \
  {                                                                  \
    if (h->NTH == 1) return xm_launch<T, R1, 1, CX>(h, H, tw, G, name); \
    if (h->NTH == 2) return xm_launch<T, R1, 2, CX>(h, H, tw, G, name); \
  }
#define XM_CASE0(T, R1) \
  if (h->NTH == 0) return xm_launch<T, R1, 0, CX>(h, H, tw, G, name);
  if (h->NX == 512) {
    XM_CASE0(128, 4) XM_CASE(128, 4)
  } else if (h->NX == 384) {
    XM_CASE0(128, 3) XM_CASE(128, 3)
  } else if (h->NX == 256) {
    // without scalars in FP64: k_xrows
    if constexpr (sizeof(CX) == 8) XM_CASE0(64, 4)
    XM_CASE(64, 4)
  } else if constexpr (sizeof(CX) == 8) {
    XM_CASE0(64, 3) XM_CASE(64, 3)
  }
#undef XM_CASE
#undef XM_CASE0
  return DG_ERR_ARG;
}

}  // namespace

bool dg_xmarch_ok(const dg_handle *h) {
  return ((h->NX == 192 && h->mixed) || h->NX == 256 || h->NX == 384 || h->NX == 512) &&
         h->NTH <= 2 && !dg_xrows_ok(h);
}

int dg_xmarch(dg_handle *h) {
  if (h->mixed)
    return xm_dispatch(h, reinterpret_cast<const float2 *>(h->H), h->twx_f,
                       reinterpret_cast<float2 *>(h->G), "k_xmarch_f32");
  return xm_dispatch(h, (const double2 *)h->H, h->twx, h->G, "k_xmarch");
}
