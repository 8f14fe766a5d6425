// The products of the periodic substep (RK_PER_1, for/periodic.f:66-215) per
// physical row: x c2r of the fields, the products u_i u_j and u_i th, x r2c.
//
// As in k_xrows (chan_xrows.cuh), NX = RF RS: RF lanes hold a row, RS points each,
// and a transform is a register step on either side of one exchange through
// shared memory.  Inverse: RF bins b + RS r of a signal (two fields) per lane, to
// [q][b]; lane q transforms its RS values into the points q + RF m.  Forward: the radix-RS
// step over the lane's points, to [p][q]; RF values of one p per lane into the bins
// p + RS m, the pair's members separated by a shuffle with the lane of the bins
// NX - k.  A signal makes 2 trips through shared memory, for 6 to 8 with Stockham
// passes between buffers, and all twiddles but the DFTs' own are W^(t i), i < RS,
// of one lane: what bound the passes was shared memory and its latency.
//
// Measured per launch, from one warp per row with those passes: FP64 256^3 368 ->
// 225 us (6 arrays of 86 x 256^2 bins written, 3 read: 812 MB at 3.6 TB/s; with 255
// registers 8 warps share an SM, and the latency of loads and FP64 bounds it), with a
// scalar 256x64x128 81 -> 52, 128^3 53 -> 31, 32^3 8.6 -> 7.4; FP32 128^3 33 -> 23,
// 96x64x96 with a scalar 25 -> 15.  The lengths with a factor 5 or 9, FP64 only, took
// a c2r launch per field, the products through physical arrays and an r2c launch
// per product: 192x64x64 with a scalar 204 -> 27 us, 100x64x64 156 -> 17.
//
// RS is 8 or more where the row is long, so that a lane's forward step feeds full
// registers; 16 x 16 at 256 points keeps every lane of the inverse's radix-16 step at
// work (32 x 8: 291 us at 256^3), except with two scalars, whose 5 x 16 points
// spill in FP64 (256x64x64: 42 against 37 us before the shifts below).  At most 128 points FP64 fits three
// CTAs per SM (128^3 with a scalar: 44 -> 40 us); above, that spills (228 -> 262).
//
// A scalar packed with U1, and the second scalar's product packed with the first's, are
// scaled to one magnitude by a power of two before the transform and back after it
// (dg_pair_shift; the largest of the planes of a warp's rows).
#include "dg_internal.cuh"
#include "fft_cols.cuh"

using namespace dgfft;

namespace {

__host__ __device__ constexpr int pr_buf(int RF, int RS, int nth) {
  const int in = ((4 + nth) / 2) * RF * (RS + 1), out = (RF / RS) * RS * (RF + 1);
  return in > out ? in : out;
}

template <int RF, int RS, int NTH, typename CX>
__global__ void __launch_bounds__(128, sizeof(CX) == 16 && RF * RS > 128 ? 2 : 3)
    k_per_rows(long nrows, const CX *__restrict__ H, long Hfield, const CX *__restrict__ tw,
               CX *__restrict__ P, long Pfield, int NZ, const unsigned *__restrict__ peak,
               int planes, int plen) {
  using TR = typename CT<CX>::T;
  constexpr int NX = RF * RS, NKXP = NX / 3 + 1, RPW = 32 / RF;
  constexpr int NF = 3 + NTH, NPIN = (NF + 1) / 2, NPROD = 6 + 3 * NTH, NPP = (NPROD + 1) / 2;
  constexpr int NB = RF / RS, NBAT = (NPP + NB - 1) / NB;
  constexpr int SI = RF * (RS + 1), SO = RS * (RF + 1), BUF = pr_buf(RF, RS, NTH);
  constexpr int KLO = NX / 3, KHI = NX - NX / 3, MO = KLO / RS + 1;
  extern __shared__ double2 sm_raw[];
  const int lane = threadIdx.x & 31, t = lane % RF;
  const bool on = 32 % RF == 0 || lane < RPW * RF;  // lanes beyond the last whole row idle along
  const int row = (threadIdx.x >> 5) * RPW + (on ? lane / RF : 0);
  CX *buf = reinterpret_cast<CX *>(sm_raw) + row * BUF;
  const long rr = (long)blockIdx.x * (4 * RPW) + row;
  const bool live = on && rr < nrows;  // a warp's rows step together
  const long ro = (rr < nrows ? rr : nrows - 1) * NKXP;
  // fields of the inverse's signal s: (U1, TH1), (U2, U3), (TH2, -)
  auto fa = [](int s) { return s < 2 ? s : 2 * s; };
  auto fb = [](int s) { return s == 0 ? 3 : s == 1 ? 2 : 2 * s + 1; };
  const CX *src = H + ro;
  // a lane's share of the peaks of U1 and the scalars on its row's plane: on their way
  // before the first bins, used behind them (96x64x96 in FP32 with a scalar: 14.7 us per
  // launch; 16.8 with the shifts ahead of the bins' loads)
  unsigned pk[1 + NTH];
  if constexpr (NTH > 0) {
    const unsigned row_c = (unsigned)(rr < nrows ? rr : nrows - 1);
    const unsigned *p = peak + (long)(row_c / (unsigned)NZ) * plen;
#pragma unroll
    for (int i = 0; i <= NTH; i++) {
      const unsigned *q = p + (long)(i ? 2 + i : 0) * planes * plen;
      pk[i] = t < plen ? __ldg(q + t) : 0;
#pragma unroll 1
      for (int l = t + RF; l < plen; l += RF) pk[i] = max(pk[i], __ldg(q + l));
    }
  }
  int d = 0, sh = 0;  // binary orders from TH1 to U1 and from TH2 to TH1
#pragma unroll
  for (int i0 = 0; i0 < NPIN * RS; i0 += RF) {
    const int i = i0 + t, s = i / RS, b = i % RS;
    const bool item = on && i < NPIN * RS;
    CX ar[RF], cr[RF];
    if (item) {
      const CX *ra = src + fa(s) * Hfield, *rb = src + fb(s) * Hfield;
      const bool two = fb(s) < NF;
#pragma unroll
      for (int r = 0; r < RF; r++) {
        // bins NX/3 + 1 .. NX - NX/3 - 1 are zero
        ar[r] = cr[r] = CT<CX>::mk(0, 0);
        if (RS * r > KLO && RS * r + RS - 1 < KHI) continue;
        const int k = b + RS * r, kk = (k <= NX / 2) ? k : NX - k;
        if (kk < NKXP) {
          ar[r] = __ldg(ra + kk);
          if (two) cr[r] = __ldg(rb + kk);
          if (kk == 0) ar[r].y = cr[r].y = 0;
        }
      }
    }
    if (NTH > 0 && i0 == 0) {
      int e[1 + NTH];
#pragma unroll
      for (int f = 0; f <= NTH; f++) e[f] = dg_mag_exp<TR>(__reduce_max_sync(0xffffffffu, pk[f]));
      d = dg_pair_shift<TR>(e[0], e[NTH > 0], 1);
      if constexpr (NTH == 2) sh = dg_pair_shift<TR>(e[1], e[2], 0);
    }
    if (item) {
      const TR sc = dg_pow2<TR>(NTH > 0 && s == 0 ? d : 0);
      CX v[RF];
#pragma unroll
      for (int r = 0; r < RF; r++) {
        const CX a = ar[r], c = cr[r];
        const int k = b + RS * r;
        v[r] = (k <= NX / 2) ? CT<CX>::mk(a.x - sc * c.y, a.y + sc * c.x)
                             : CT<CX>::mk(a.x + sc * c.y, sc * c.x - a.y);
      }
      dft<RF>(v, +1);
      CX *o = buf + s * SI + b;
#pragma unroll
      for (int q = 0; q < RF; q++) o[q * (RS + 1)] = v[q];
    }
  }
  __syncwarp();
  CX w[RS];  // W^(t i)
#pragma unroll
  for (int i = 1; i < RS; i++) w[i] = __ldg(tw + t * i);
  TR u[NF][RS];
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
      u[fa(s)][m] = v[m].x;
      if (fb(s) < NF) u[fb(s)][m] = NTH > 0 && s == 0 ? v[m].y * dg_pow2<TR>(-d) : v[m].y;
    }
  }
  __syncwarp();
  // product i: U1U1 U1U2 U1U3 U2U2 U2U3 U3U3, then U_j TH_n
  auto prod = [&](int i, int m) -> TR {
    if (i >= NPROD) return (TR)0;
    const int a = i < 6 ? (i < 3 ? 0 : i < 5 ? 1 : 2) : (i - 6) % 3;
    const int b = i < 6 ? (i < 3 ? i : i < 5 ? i - 2 : 2) : 3 + (i - 6) / 3;
    return u[a][m] * u[b < NF ? b : 0][m];
  };
#pragma unroll
  for (int bt = 0; bt < NBAT; bt++) {
    const int s0 = bt * NB;
#pragma unroll
    for (int sl = 0; sl < NB; sl++) {
      if (s0 + sl >= NPP) continue;
      CX v[RS];
#pragma unroll
      for (int m = 0; m < RS; m++) {
        v[m] = CT<CX>::mk(prod(2 * (s0 + sl), m), prod(2 * (s0 + sl) + 1, m));
        if (NTH == 2 && s0 + sl == 4) v[m].y *= dg_pow2<TR>(sh);  // (U3 TH1, U1 TH2)
      }
      dft<RS>(v, -1);
#pragma unroll
      for (int p = 0; p < RS; p++)
        if (on) buf[sl * SO + p * (RF + 1) + t] = p > 0 ? cmul(v[p], w[p]) : v[p];
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
    CX *o = P + 2 * (s0 + sl) * Pfield + ro;
    const bool two = 2 * (s0 + sl) + 1 < NPROD;
    constexpr TR hx = (TR)(0.5 / (double)NX);
#pragma unroll
    for (int m = 0; m < MO; m++) {
      CX zm = CT<CX>::mk(__shfl_sync(0xffffffffu, v[RF - 1 - m].x, other),
                         __shfl_sync(0xffffffffu, v[RF - 1 - m].y, other));
      if (p == 0) zm = v[(RF - m) % RF];
      const int k = p + RS * m;
      if (!item || !live || k >= NKXP) continue;
      const CX zk = v[m];
      // A = (Z_k + conj Z_{N-k})/2, B = -i/2 (Z_k - conj Z_{N-k}), over NX
      o[k] = CT<CX>::mk(hx * (zk.x + zm.x), hx * (zk.y - zm.y));
      TR hb = hx;
      if constexpr (NTH == 2) {
        if (s0 + sl == 4) hb *= dg_pow2<TR>(-sh);
      }
      if (two) o[Pfield + k] = CT<CX>::mk(hb * (zk.y + zm.y), -hb * (zk.x - zm.x));
    }
    __syncwarp();
  }
}

template <int RF, int RS, int NTH, typename CX>
int pr_launch(dg_handle *h, const CX *H, const CX *tw, CX *P, const char *name) {
  auto kern = k_per_rows<RF, RS, NTH, CX>;
  dg_big_smem((const void *)kern);
  const long nrows = (long)h->NY * h->NZ, pf = nrows * h->nkxp;
  constexpr int rows = 4 * (32 / RF);
  dg_kt_begin(h, name, h->st);
  kern<<<dg_cdiv(nrows, rows), 128, sizeof(CX) * rows * (size_t)pr_buf(RF, RS, NTH), h->st>>>(
      nrows, H, pf, tw, P, pf, h->NZ, h->peak, h->NY, h->peak_len);
  DG_LAUNCHED();
  return DG_OK;
}

template <int RF, int RS, typename CX>
int pr_th(dg_handle *h, const CX *H, const CX *tw, CX *P, const char *name) {
  if (h->NTH == 0) return pr_launch<RF, RS, 0, CX>(h, H, tw, P, name);
  if (h->NTH == 1) return pr_launch<RF, RS, 1, CX>(h, H, tw, P, name);
  if constexpr (RS == 16) return DG_ERR_ARG;  // 256 points with two scalars: see above
  else return pr_launch<RF, RS, 2, CX>(h, H, tw, P, name);
}

}  // namespace

// what dg_per_rows has an instance for: in FP32 the lengths that dg_per_mixed_ok admits,
// in FP64 further ones
bool dg_per_rows_ok(int nx, int nth, bool mixed) {
  if (mixed) return dg_per_mixed_ok(nx, nth);
  if (nth > 2) return false;
  switch (nx) {
    case 16: case 32: case 48: case 64: case 96: case 128: case 256: case 20: case 24: case 30:
    case 36: case 40: case 50: case 54: case 60: case 72: case 80: case 90: case 100: case 108: case 120:
    case 144: case 150: case 160: case 162: case 180: case 192: case 200: case 216: case 240:
    case 270: case 288: case 320: return true;
    default: return false;
  }
}

int dg_per_rows(dg_handle *h) {
#define PR(N, RF, RS, CX, TW, NAME)                                                           \
  case N:                                                                                     \
    return pr_th<RF, RS, CX>(h, reinterpret_cast<const CX *>(h->H), (const CX *)TW,           \
                             reinterpret_cast<CX *>(h->P), NAME);
#define PR_BOTH(CX, TW, NAME)                                                                 \
  PR(16, 4, 4, CX, TW, NAME) PR(32, 8, 4, CX, TW, NAME) PR(48, 8, 6, CX, TW, NAME)            \
  PR(64, 8, 8, CX, TW, NAME) PR(96, 16, 6, CX, TW, NAME) PR(128, 16, 8, CX, TW, NAME)         \
  case 256:                                                                                   \
    if (h->NTH == 2)                                                                          \
      return pr_launch<32, 8, 2, CX>(h, reinterpret_cast<const CX *>(h->H), (const CX *)TW,   \
                                     reinterpret_cast<CX *>(h->P), NAME);                     \
    return pr_th<16, 16, CX>(h, reinterpret_cast<const CX *>(h->H), (const CX *)TW,           \
                             reinterpret_cast<CX *>(h->P), NAME);
  if (h->mixed) {
    switch (h->NX) {
      PR_BOTH(float2, h->twx_f, "k_per_rows_f32")
      default: return DG_ERR_ARG;
    }
  }
  switch (h->NX) {
    PR_BOTH(double2, h->twx, "k_per_rows")
#define P64(N, RF, RS) PR(N, RF, RS, double2, h->twx, "k_per_rows")
    P64(20, 5, 4) P64(24, 6, 4) P64(30, 6, 5) P64(36, 9, 4) P64(40, 8, 5) P64(54, 9, 6) P64(60, 10, 6)
    P64(72, 9, 8) P64(80, 16, 5) P64(90, 15, 6) P64(100, 20, 5) P64(108, 18, 6) P64(120, 15, 8)
    P64(144, 16, 9) P64(160, 16, 10) P64(180, 15, 12) P64(192, 16, 12)
    P64(200, 20, 10) P64(216, 24, 9) P64(240, 16, 15) P64(50, 10, 5)
    P64(150, 30, 5) P64(162, 18, 9) P64(270, 30, 9) P64(288, 32, 9) P64(320, 32, 10)
    default: return DG_ERR_ARG;
  }
}
