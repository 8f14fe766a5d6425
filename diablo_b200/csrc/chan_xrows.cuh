// The x-row stage of a channel substep for the short row lengths: x c2r of
// every field, the products of for/channel.f:409-571,665-720 and their x r2c, a
// group of RF lanes per z-row marching up through a chunk of planes.
//
// With NX = RF RS a transform is two register transforms with one exchange through
// shared memory between them.  Inverse: a lane takes the RF bins b + RS r of a
// signal (two fields packed) from global memory, transforms them and leaves them at [q][b];
// lane q takes its RS values, times W_N^(-b q), and transforms them into the
// points x = q + RF m, m = 0..RS-1, of every field.  Those are the inputs of the forward's first
// step, whose index runs over m: the products go from the lane's registers into a radix-RS
// transform, times W_N^(q p), to [p][q]; a lane then transforms the RF
// values of one p into the bins p + RS m.  The twiddles W_N^(q i) are RS - 1
// constants of the lane in both directions, and the bins that a pair's two members are
// separated with, k and NX - k, lie in two lanes of a signal: a shuffle.  Rows need no CTA barrier.
//
// A row and plane makes 2 trips through shared memory per inverse signal and 2 (and
// the shuffles) per forward one, where passes between buffers (input, two
// passes, output) made 6 each; that bandwidth bounded the stage (60% of its
// peak), which one warp per row with Stockham passes took 73 us for at
// 128x129x128 and now takes 55 (events around eager launches): 29 -> 17 us at 128x65x32
// with a scalar, 79 -> 31 at 96x65x96, 75 -> 47 at 64x129x128 with two; FP32
// 59 -> 49 at 128x129x128.  Two CTAs per SM at up to 255 registers: a lane's points of two
// planes and its RF values are registers (with 168 and spills 60 us; FP32
// without scalars fits 168 and three CTAs, 49 us against 55).
//
// The pairs are those of k_xprod (chan_kernels.cu), as in k_xmarch; forward
// signals go through in batches of NB = RF / RS, one item per lane.  Members that
// have different units are brought to one magnitude by a power of two before a transform
// and back after it (dg_pair_shift): a scalar packed with U1, the second scalar
// packed with the first (0 to 6% per launch with scalars: 30.4 -> 30.8 us at 96x65x96
// with one, 124 -> 132 at 320x65x48 with two).
#pragma once

#include <math.h>

#include "dg_internal.cuh"
#include "fft_cols.cuh"

using namespace dgfft;

namespace {

struct XrArgs {
  int NZ;
  long Hfield, Gfield;
  int chunk, jbase, jtop;
  const double *dyf, *dy, *kx;
  const unsigned *peak;  // of H's planes
  int planes, plen;
};

__host__ __device__ constexpr int xr_pairs(int nth) { return 4 + nth + (nth + 1) / 2; }
// fields of the inverse's signal s, as in k_xmarch: (U1, TH1), (U2, U3), (TH2, -)
__host__ __device__ constexpr int xr_fa(int s) { return s < 2 ? s : 2 * s; }
__host__ __device__ constexpr int xr_fb(int s) { return s == 0 ? 3 : s == 1 ? 2 : 2 * s + 1; }
// arrays of G that pair s writes: A (-1: none), and B or the flux -i kx A - c B
__host__ __device__ constexpr int xr_ga(int s, int nth) {
  return s == 0 ? 0 : s == 3 ? 2 : s >= 4 + nth ? 6 + 4 * (s - 4 - nth) : -1;
}
__host__ __device__ constexpr int xr_gb(int s, int nth) {
  return s == 0 ? 5 : s == 1 ? 1 : s == 2 ? 3 : s == 3 ? 4 : s < 4 + nth ? 7 + 2 * (s - 4)
         : (2 * (s - 4 - nth) + 1 < nth ? 8 + 4 * (s - 4 - nth) : -1);
}
__host__ __device__ constexpr bool xr_flux(int s, int nth) { return s < 3 || (s >= 4 && s < 4 + nth); }

// bank spread: [q][b] and [p][q] with one slot between rows
__host__ __device__ constexpr int xr_buf(int RF, int RS, int nth) {
  const int in = ((4 + nth) / 2) * RF * (RS + 1), out = (RF / RS) * RS * (RF + 1);
  return in > out ? in : out;
}

template <int RF, int RS, int NTH, typename CX>
__global__ void __launch_bounds__(128, sizeof(CX) == 8 && NTH == 0 ? 3 : 2)
    k_xrows(XrArgs A, const CX *__restrict__ H, const CX *__restrict__ tw, CX *__restrict__ G) {
  using TR = typename CT<CX>::T;
  constexpr bool F32 = sizeof(TR) == 4;
  constexpr int NX = RF * RS, NKXP = NX / 3 + 1, RPW = 32 / RF;  // rows per warp
  constexpr int NF = 3 + NTH, NPIN = (NF + 1) / 2, NPP = xr_pairs(NTH);
  static_assert(!F32 || 32 % RF == 0, "the FP32 means are summed over whole groups of lanes");
  constexpr int NB = RF / RS, NBAT = (NPP + NB - 1) / NB;
  constexpr int SI = RF * (RS + 1), SO = RS * (RF + 1), BUF = xr_buf(RF, RS, NTH);
  constexpr int KLO = NX / 3, KHI = NX - NX / 3, MO = KLO / RS + 1;
  extern __shared__ double2 sm_raw[];
  const int lane = threadIdx.x & 31, t = lane % RF;
  const bool on = 32 % RF == 0 || lane < RPW * RF;  // lanes beyond the last whole row idle along
  const int row = (threadIdx.x >> 5) * RPW + (on ? lane / RF : 0);
  constexpr int rows = (128 / 32) * RPW;
  CX *buf = reinterpret_cast<CX *>(sm_raw) + row * BUF;
  TR *prv = reinterpret_cast<TR *>(reinterpret_cast<CX *>(sm_raw) + rows * BUF) + row * (NF * NX);
  int *shf = reinterpret_cast<int *>(
      reinterpret_cast<TR *>(reinterpret_cast<CX *>(sm_raw) + rows * BUF) + rows * (NF * NX));
  const int NZ = A.NZ, zr = blockIdx.x * rows + row;
  const bool live = on && zr < NZ;  // a warp's rows step together
  const int z = zr < NZ ? zr : NZ - 1;
  CX w[RS];
#pragma unroll
  for (int i = 1; i < RS; i++) w[i] = tw[t * i];
  const int j0 = A.jbase + blockIdx.y * A.chunk;
  const int j1 = min(j0 + A.chunk - 1, A.jtop);
  const long plane = (long)NZ * NKXP;
  const CX *Hz = H + (long)z * NKXP;
  dg_pdl_wait();  // H comes from the z inverse

  TR cur[NF][RS], nxt[NF][RS];
  double dcur[NF], dnxt[NF], dprv[NF];  // row means (FP32 form)

  if constexpr (NTH > 0)
    dg_plane_shifts<TR, NTH>(shf, A.peak, A.planes, A.plen, j0 - 1, j1 - j0 + 3);
  int shc = 0, shn = 0;  // two scalars: TH2's shift to TH1 in their common pair, planes j and j+1
  auto load_plane = [&](int pl, TR (&dst)[NF][RS], double (&dcv)[NF], int &sh) {
    const CX *src = Hz + (long)pl * plane;
    const int sw = NTH > 0 ? shf[pl - j0 + 1] : 0, d = (short)sw;  // TH1 goes times 2^d
    if constexpr (F32) {
#pragma unroll
      for (int f = 0; f < NF; f++) dcv[f] = (double)__ldg(src + f * A.Hfield).x;
    }
    if constexpr (NTH == 2) {
      if constexpr (F32)  // the products hold the row means, the peaks do not
        sh = dg_pair_shift<TR>(max((sw >> 24) & 255, dg_mag_exp<TR>(dg_mag((TR)dcv[3]))),
                               max((sw >> 16) & 255, dg_mag_exp<TR>(dg_mag((TR)dcv[4]))), 0);
      else
        sh = sw >> 16;
    }
#pragma unroll
    for (int i0 = 0; i0 < NPIN * RS; i0 += RF) {
      const int i = i0 + t, s = i / RS, b = i % RS;
      if (on && i < NPIN * RS) {
        const CX *ra = src + xr_fa(s) * A.Hfield, *rb = src + xr_fb(s) * A.Hfield;
        const bool two = xr_fb(s) < NF;
        const TR sc = dg_pow2<TR>(NTH > 0 && s == 0 ? d : 0);
        CX v[RF];
#pragma unroll
        for (int r = 0; r < RF; r++) {
          // bins NX/3 + 1 .. NX - NX/3 - 1 are zero
          v[r] = CT<CX>::mk(0, 0);
          if (RS * r > KLO && RS * r + RS - 1 < KHI) continue;
          const int k = b + RS * r, kk = (k <= NX / 2) ? k : NX - k;
          CX a = CT<CX>::mk(0, 0), c = CT<CX>::mk(0, 0);
          if (kk < NKXP && !(F32 && kk == 0)) {
            a = __ldg(ra + kk);
            if (two) c = __ldg(rb + kk);
            if (kk == 0) a.y = c.y = 0;
          }
          v[r] = (k == kk) ? CT<CX>::mk(a.x - sc * c.y, a.y + sc * c.x)
                           : CT<CX>::mk(a.x + sc * c.y, sc * c.x - a.y);
        }
        dft<RF>(v, +1);
        CX *o = buf + s * SI + b;
#pragma unroll
        for (int q = 0; q < RF; q++) o[q * (RS + 1)] = v[q];
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NPIN; s++) {
      CX v[RS];
#pragma unroll
      for (int b = 0; b < RS; b++) {
        v[b] = buf[s * SI + t * (RS + 1) + b];
        if (b > 0) v[b] = cmul(v[b], conjg(w[b]));
      }
      dft<RS>(v, +1);
#pragma unroll
      for (int m = 0; m < RS; m++) {
        dst[xr_fa(s)][m] = v[m].x;
        if (xr_fb(s) < NF)
          dst[xr_fb(s)][m] = s == 0 ? v[m].y * dg_pow2<TR>(-d) : v[m].y;
      }
    }
    __syncwarp();
  };

  load_plane(j0 - 1, cur, dprv, shc);
#pragma unroll
  for (int f = 0; f < NF; f++)
#pragma unroll
    for (int m = 0; m < RS; m++)
      if (on) prv[(f * RS + m) * RF + t] = cur[f][m];
  load_plane(j0, cur, dcur, shc);
#pragma unroll 1
  for (int j = j0; j <= j1; j++) {
    load_plane(j + 1, nxt, dnxt, shn);
    const double dyfj = A.dyf[j], dyfm = A.dyf[j - 1], wgyd = 1.0 / (2.0 * A.dy[j]);
    const double id2 = 1.0 / (2.0 * dyfj), idyj = 1.0 / A.dy[j];
    const TR cj = (TR)(dyfj * wgyd), cm = (TR)(dyfm * wgyd);
    auto old = [&](int f, int m) -> TR { return prv[(f * RS + m) * RF + t]; };
    double acc[2 * NB] = {};  // FP32 form: sums of the products of the fluctuations
    // FP32 form: (D1 + a)(D2 + b) without its mean part D1 D2; the sum of a b
    // goes to accumulator i in FP64
    auto pr = [&](double d1, TR a, double d2, TR b, int i, double sg) -> TR {
      if constexpr (F32) acc[i] = fma(sg * (double)a, (double)b, acc[i]);
      return (TR)sg * ((TR)d1 * b + (TR)d2 * a + a * b);
    };
    // (X(j+1) + X(j)) U2(j+1) - (X(j) + X(j-1)) U2(j)
    auto rise = [&](int f, int m, int i) -> TR {
      const TR x = cur[f][m], xp = nxt[f][m] + x, xm = x + old(f, m);
      if constexpr (F32)
        return pr(dnxt[f] + dcur[f], xp, dnxt[1], nxt[1][m], i, 1.0) +
               pr(dcur[f] + dprv[f], xm, dcur[1], cur[1][m], i, -1.0);
      else
        return xp * nxt[1][m] - xm * cur[1][m];
    };
    // F(f) F(g) at plane j
    auto prod = [&](int f, int g, int m, int i) -> TR {
      if constexpr (F32) return pr(dcur[f], cur[f][m], dcur[g], cur[g][m], i, 1.0);
      else return cur[f][m] * cur[g][m];
    };
    // Ubar U2 at GY j
    auto ubar = [&](int f, int m, int i) -> TR {
      const TR x = cj * cur[f][m] + cm * old(f, m);
      if constexpr (F32)
        return pr((dyfj * dcur[f] + dyfm * dprv[f]) * wgyd, x, dcur[1], cur[1][m], i, 1.0);
      else
        return x * cur[1][m];
    };
    auto pair_at = [&](int s, int m, int i) -> CX {
      if (s == 0) return CT<CX>::mk(prod(2, 0, m, i), rise(2, m, i + 1));
      if (s == 1) return CT<CX>::mk(prod(0, 0, m, i), rise(0, m, i + 1));
      if (s == 2) {
        const TR gp = (TR)0.5 * (cur[1][m] + nxt[1][m]), gm = (TR)0.5 * (old(1, m) + cur[1][m]);
        TR b;
        if constexpr (F32) {
          const double gpd = 0.5 * (dcur[1] + dnxt[1]), gmd = 0.5 * (dprv[1] + dcur[1]);
          b = pr(gpd, gp, gpd, gp, i + 1, 1.0) + pr(gmd, gm, gmd, gm, i + 1, -1.0);
        } else {
          b = gp * gp - gm * gm;
        }
        return CT<CX>::mk(ubar(0, m, i), b);
      }
      if (s == 3) return CT<CX>::mk(ubar(2, m, i), prod(2, 2, m, i + 1));
      if (s < 4 + NTH) {
        const int f = s - 1 < NF ? s - 1 : 0;
        return CT<CX>::mk(prod(f, 0, m, i), rise(f, m, i + 1));
      }
      const int n = 2 * (s - 4 - NTH), f = 3 + n < NF ? 3 + n : 0, g = 4 + n < NF ? 4 + n : 0;
      return CT<CX>::mk(prod(f, 2, m, i),
                        n + 1 < NTH ? dg_pow2<TR>(shc) * prod(g, 2, m, i + 1) : (TR)0);
    };
    // mean parts of the pair's products
    auto means = [&](int s, double &da, double &db) {
      const double *c = dcur, *n = dnxt, *p = dprv;
      db = 0.0;
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
        const int f = s - 1 < NF ? s - 1 : 0;
        da = c[f] * c[0];
        db = (n[f] + c[f]) * n[1] - (c[f] + p[f]) * c[1];
      } else {
        const int i = 2 * (s - 4 - NTH), f = 3 + i < NF ? 3 + i : 0, g = 4 + i < NF ? 4 + i : 0;
        da = c[f] * c[2];
        if (i + 1 < NTH) db = c[g] * c[2];
      }
    };
#pragma unroll
    for (int bt = 0; bt < NBAT; bt++) {
      const int s0 = bt * NB;
      // the pairs at the lane's points, the radix-RS step, to [p][q]
      if constexpr (F32) {
#pragma unroll
        for (int i = 0; i < 2 * NB; i++) acc[i] = 0.0;
      }
#pragma unroll
      for (int sl = 0; sl < NB; sl++) {
        if (s0 + sl >= NPP) continue;
        CX v[RS];
#pragma unroll
        for (int m = 0; m < RS; m++) v[m] = pair_at(s0 + sl, m, 2 * sl);
        dft<RS>(v, -1);
#pragma unroll
        for (int p = 0; p < RS; p++)
          if (on) buf[sl * SO + p * (RF + 1) + t] = p > 0 ? cmul(v[p], w[p]) : v[p];
      }
      if constexpr (F32) {
#pragma unroll
        for (int i = 0; i < 2 * NB; i++)
#pragma unroll
          for (int o = RF / 2; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
      }
      __syncwarp();
      // the bins p + RS m of signal s0 + sl
      const int sl = NB > 1 ? t / RS : 0, p = t % RS;
      const bool item = on && t < NB * RS && s0 + sl < NPP;
      CX v[RF];
#pragma unroll
      for (int b = 0; b < RF; b++) v[b] = item ? buf[sl * SO + p * (RF + 1) + b] : CT<CX>::mk(0, 0);
      dft<RF>(v, -1);
      const int other = lane - t + (t < NB * RS ? sl * RS + (p ? RS - p : 0) : t);
      int ga = xr_ga(s0, NTH), gb = xr_gb(s0, NTH);
      bool fl = xr_flux(s0, NTH);
      double cf = s0 == 2 ? idyj : id2;
#pragma unroll
      for (int i = 1; i < NB; i++)
        if (sl == i && s0 + i < NPP) {
          ga = xr_ga(s0 + i, NTH);
          gb = xr_gb(s0 + i, NTH);
          fl = xr_flux(s0 + i, NTH);
          cf = s0 + i == 2 ? idyj : id2;
        }
      CX *o = G + (long)j * plane + (long)z * NKXP;
      constexpr double hx = 0.5 / (double)NX;
#pragma unroll
      for (int m = 0; m < MO; m++) {
        CX zm = CT<CX>::mk(__shfl_sync(0xffffffffu, v[RF - 1 - m].x, other),
                           __shfl_sync(0xffffffffu, v[RF - 1 - m].y, other));
        if (p == 0) zm = v[(RF - m) % RF];
        const int k = p + RS * m;
        if (!item || !live || k >= NKXP) continue;
        const CX zk = v[m];
        // the pair's members, scaled by 1/NX: A = (Z_k + conj Z_{N-k})/2,
        // B = -i/2 (Z_k - conj Z_{N-k})
        double2 a = make_double2(hx * ((double)zk.x + zm.x), hx * ((double)zk.y - zm.y));
        double2 b = make_double2(hx * ((double)zk.y + zm.y), -hx * ((double)zk.x - zm.x));
        if constexpr (NTH == 2) {
          if (s0 + sl == 4 + NTH) {
            b.x *= dg_pow2<double>(-shc);
            b.y *= dg_pow2<double>(-shc);
          }
        }
        if constexpr (F32) {
          if (m == 0 && k == 0) {
            double da = 0.0, db = 0.0;
#pragma unroll
            for (int i = 0; i < NB; i++)
              if (sl == i && s0 + i < NPP) {
                means(s0 + i, da, db);
                a = make_double2(da + acc[2 * i] / (double)NX, 0.0);
                b = make_double2(db + acc[2 * i + 1] / (double)NX, 0.0);
              }
          }
        }
        if (ga >= 0) o[ga * A.Gfield + k] = CT<CX>::mk((TR)a.x, (TR)a.y);
        if (gb >= 0) {
          const double KX = A.kx[k];
          const double fx = fl ? KX * a.y - b.x * cf : b.x, fy = fl ? -KX * a.x - b.y * cf : b.y;
          o[gb * A.Gfield + k] = CT<CX>::mk((TR)fx, (TR)fy);
        }
      }
      __syncwarp();
    }
    // plane j becomes j-1, j+1 becomes j
    shc = shn;
#pragma unroll
    for (int f = 0; f < NF; f++) {
#pragma unroll
      for (int m = 0; m < RS; m++) {
        if (on) prv[(f * RS + m) * RF + t] = cur[f][m];
        cur[f][m] = nxt[f][m];
      }
      if constexpr (F32) {
        dprv[f] = dcur[f];
        dcur[f] = dnxt[f];
      }
    }
  }
}

template <int RF, int RS, int NTH, typename CX>
int xr_launch(dg_handle *h, int ja, int jb, const CX *H, const CX *tw, CX *G, const char *name) {
  auto kern = k_xrows<RF, RS, NTH, CX>;
  dg_big_smem((const void *)kern);
  XrArgs A;
  A.NZ = h->NZ;
  A.Hfield = A.Gfield = (long)h->nplanes * h->NZ * h->nkxp;
  A.jbase = ja; A.jtop = jb;
  A.dyf = h->dyf; A.dy = h->dy; A.kx = h->kx;
  A.peak = h->peak; A.planes = h->NY + 2; A.plen = h->peak_len;
  constexpr int rows = 4 * (32 / RF);
  const size_t sm = sizeof(CX) * rows * (size_t)xr_buf(RF, RS, NTH) +
                    sizeof(typename CT<CX>::T) * rows * (3 + NTH) * (size_t)(RF * RS) +
                    (NTH > 0 ? sizeof(int) * (h->NY + 2) : 0);
  const int nplan = jb - ja + 1, zb = dg_cdiv(h->NZ, rows);
  A.chunk = h->xrow_chunk > 0 ? (h->xrow_chunk < nplan ? h->xrow_chunk : nplan)
                              : dg_march_chunk(nplan, zb, (const void *)kern, 128, sm, 1.0, 0.7);
  dg_kt_begin(h, name, h->st);
  DG_CUDA(dg_launch(h->pdl, kern, dim3(zb, dg_cdiv(nplan, A.chunk)), dim3(128), sm, h->st, A, H, tw,
                    G));
  DG_LAUNCHED();
  return DG_OK;
}

template <int RF, int RS, typename CX>
int xr_th(dg_handle *h, int ja, int jb, const CX *H, const CX *tw, CX *G, const char *name) {
  if (h->NTH == 0) return xr_launch<RF, RS, 0, CX>(h, ja, jb, H, tw, G, name);
  if (h->NTH == 1) return xr_launch<RF, RS, 1, CX>(h, ja, jb, H, tw, G, name);
  return xr_launch<RF, RS, 2, CX>(h, ja, jb, H, tw, G, name);
}

}  // namespace
