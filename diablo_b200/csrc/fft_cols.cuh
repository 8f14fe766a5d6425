// Transforms of columns (z, and y of the periodic box) that exchange data
// through shared memory once, or twice for the long ones.
//
// A CTA takes KXG neighbouring columns of one plane.  With N = RA RB, input
// index n = b + RB r and output index o = q + RA m,
//   X(o) = sum_b W_RB^(b m) W_N^(b q) sum_r x(b + RB r) W_RA^(r q):
// a thread loads the RA inputs of one (column, b) straight from global memory,
// transforms them in registers, multiplies by W_N^(b q) and leaves them at [q][b]
// in shared memory; after one barrier a thread takes the RB values of one (column, q),
// transforms them in registers and stores its outputs.  Lengths above 256
// are N = RA RB RC: the RB RC transform of each q runs the same way, the
// radix-RB step in place (a thread's reads and writes are the same slots).
// Neighbouring lanes hold neighbouring columns everywhere, so global accesses
// are whole 128-byte row segments and shared memory has no bank conflicts.
//
// Bound by HBM and latency (16 warps per SM, 16 loads in flight per thread).
// Against the Stockham passes in shared memory (input, two or three passes and output each a
// trip through it): inverse 27 -> 21 us at 128x129x128 (3 fields), 761 -> 511 us at 512x257x384 (4);
// z forward 38 -> 31 and 267 -> 73 us (324 points, 74 planes, 4 fields: run-time radices); periodic
// 256^3 107 -> 75 us (inverse) and 186 -> 150 us (forward, 6 products).
#pragma once

#include "dg_internal.cuh"
#include "fft.cuh"

namespace dgfft {

// Prime-factor DFTs (no twiddles between the factors), R = P Q: inputs
// n = (Q n1 + P n2) mod R, outputs k = (e1 k1 + e2 k2) mod R with e1 = 1 mod P, 0 mod Q and
// e2 = 0 mod P, 1 mod Q.
template <int P, int Q, int E1, int E2> struct DFTpf {
  template <typename C> static __device__ __forceinline__ void run(C *v, int sign) {
    constexpr int R = P * Q;
    C a[Q][P];
#pragma unroll
    for (int n2 = 0; n2 < Q; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < P; n1++) a[n2][n1] = v[(Q * n1 + P * n2) % R];
      DFT<P>::run(a[n2], sign);
    }
#pragma unroll
    for (int k1 = 0; k1 < P; k1++) {
      C t[Q];
#pragma unroll
      for (int n2 = 0; n2 < Q; n2++) t[n2] = a[n2][k1];
      DFT<Q>::run(t, sign);
#pragma unroll
      for (int k2 = 0; k2 < Q; k2++) v[(E1 * k1 + E2 * k2) % R] = t[k2];
    }
  }
};
template <> struct DFT<6> : DFTpf<2, 3, 3, 4> {};
template <> struct DFT<10> : DFTpf<2, 5, 5, 6> {};
template <> struct DFT<12> : DFTpf<4, 3, 9, 4> {};
template <> struct DFT<15> : DFTpf<3, 5, 10, 6> {};
template <> struct DFT<20> : DFTpf<4, 5, 5, 16> {};

// 9-point DFT as 3 x 3: n = 3 n1 + n2, k = k1 + 3 k2, twiddles exp(sign 2 pi i m / 9)
template <> struct DFT<9> {
  template <typename C> static __device__ __forceinline__ void run(C *v, int sign) {
    using T = typename CT<C>::T;
    const T Cs[5] = {(T)1.0, (T)0.76604444311897803520, (T)0.17364817766693034885, (T)-0.5,
                     (T)-0.93969262078590838405};
    const T Sn[5] = {(T)0.0, (T)0.64278760968653932632, (T)0.98480775301220805937,
                     (T)0.86602540378443864676, (T)0.34202014332566873304};
    C a[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++) {
      C t[3] = {v[n2], v[3 + n2], v[6 + n2]};
      DFT<3>::run(t, sign);
#pragma unroll
      for (int k1 = 0; k1 < 3; k1++) {
        const int m = n2 * k1;
        a[n2][k1] = m ? cmul(t[k1], CT<C>::mk(Cs[m], sign * Sn[m])) : t[k1];
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
      C t[3] = {a[0][k1], a[1][k1], a[2][k1]};
      DFT<3>::run(t, sign);
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) v[k1 + 3 * k2] = t[k2];
    }
  }
};

template <> struct DFT<18> : DFTpf<2, 9, 9, 10> {};
template <> struct DFT<24> : DFTpf<3, 8, 16, 9> {};
template <> struct DFT<30> : DFTpf<5, 6, 6, 25> {};

// 32-point DFT as 4 x 8: n = 8 n1 + n2, k = k1 + 4 k2, twiddles exp(sign 2 pi i m / 32)
template <> struct DFT<32> {
  template <typename C> static __device__ __forceinline__ void run(C *v, int sign) {
    using T = typename CT<C>::T;
    // cos(2 pi m / 32), m = 0..24; sin(2 pi m / 32) = cos(2 pi (m - 8) / 32)
    const T Q[9] = {(T)1.0, (T)0.98078528040323044913, (T)0.92387953251128675613,
                    (T)0.83146961230254523708, (T)0.70710678118654752440, (T)0.55557023301960222474,
                    (T)0.38268343236508977173, (T)0.19509032201612826785, (T)0.0};
    C a[8][4];
#pragma unroll
    for (int n2 = 0; n2 < 8; n2++) {
      C t[4] = {v[n2], v[8 + n2], v[16 + n2], v[24 + n2]};
      DFT<4>::run(t, sign);
#pragma unroll
      for (int k1 = 0; k1 < 4; k1++) {
        const int m = n2 * k1;  // 0..21
        const T cs = m <= 8 ? Q[m] : m <= 16 ? -Q[16 - m] : -Q[m - 16];
        const T sn = m <= 8 ? Q[8 - m] : m <= 16 ? Q[m - 8] : -Q[24 - m];
        a[n2][k1] = m ? cmul(t[k1], CT<C>::mk(cs, sign * sn)) : t[k1];
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      C t[8];
#pragma unroll
      for (int n2 = 0; n2 < 8; n2++) t[n2] = a[n2][k1];
      DFT<8>::run(t, sign);
#pragma unroll
      for (int k2 = 0; k2 < 8; k2++) v[k1 + 4 * k2] = t[k2];
    }
  }
};

// The split of a column length; rc = 1: two steps.
struct ColPlan {
  int n, ra, rb, rc;
};

// compile-time lengths
__host__ __device__ constexpr int cols_ra(int n) {
  return n == 16 ? 4 : n == 32 ? 4 : n == 48 ? 6 : n == 64 ? 8 : n == 96 ? 12 : n == 128 ? 16
         : n == 192 ? 12 : n == 256 ? 16 : n == 384 ? 8 : n == 512 ? 8 : 0;
}
__host__ __device__ constexpr int cols_rc(int n) { return n == 384 ? 6 : n == 512 ? 8 : 1; }
__host__ __device__ constexpr int cols_rb(int n) { return n / (cols_ra(n) * cols_rc(n)); }

// columns per CTA: 16 up to 128 points, 8 above (32 KB of shared memory at
// 128 and 256 points in FP64)
__host__ __device__ constexpr int cols_log_kxg(int n) {
  return n <= 128 ? 4 : n <= 512 ? 3 : n <= 1024 ? 2 : 1;
}
constexpr int COLS_THR = 128;

// run-time split of n: two factors up to 256, else three, out of the radices
// below, the largest as small as possible (registers).  False: no such split.
static inline bool cols_plan(int n, ColPlan *pl) {
  static const int radix[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16};
  int best = 1 << 30;
  for (int a : radix)
    for (int b : radix) {
      if (n % (a * b)) continue;
      const int c = n / (a * b);
      if (c != 1) {
        bool ok = false;
        for (int r : radix) ok = ok || r == c;
        if (!ok) continue;
      }
      // two steps before three; then the smaller largest radix; then the
      // larger first one (loads in flight)
      const int big = a > b ? (a > c ? a : c) : (b > c ? b : c);
      const int cost = (c == 1 ? 0 : 10000) + big * 100 - a;
      if (cost < best) {
        best = cost;
        *pl = {n, a, b, c};
      }
    }
  return best < (1 << 30) && n <= 1024;
}

#if defined(__CUDACC__)
// 1. radix-R transforms of the inputs n = b + nb r, twiddled, to sm[(q nb + b) KXG + c];
// tw: exp(-2 pi i m / N)
template <int R, int SIGN, typename CX, typename Load>
__device__ __forceinline__ void cols_first(CX *__restrict__ sm, int nb, int lk,
                                           const CX *__restrict__ tw, Load load) {
#pragma unroll 1
  for (int i = threadIdx.x; i < nb << lk; i += COLS_THR) {
    const int c = i & ((1 << lk) - 1), b = i >> lk;
    CX v[R];
    load.template get<R>(v, b, nb, c);
    dft<R>(v, SIGN);
#pragma unroll
    for (int q = 0; q < R; q++) {
      if (q > 0) {
        CX t = __ldg(tw + b * q);
        if (SIGN > 0) t.y = -t.y;
        v[q] = cmul(v[q], t);
      }
      sm[((q * nb + b) << lk) + c] = v[q];
    }
  }
}

// 2. (three steps only) radix R over r2 of b = b2 + rc r2 for every q, twiddled
// by W_(R rc)^(b2 q2) = tw[b2 q2 ra], in place
template <int R, int SIGN, typename CX>
__device__ __forceinline__ void cols_mid(CX *__restrict__ sm, int ra, int rc, int lk,
                                         const CX *__restrict__ tw) {
#pragma unroll 1
  for (int i = threadIdx.x; i < (ra * rc) << lk; i += COLS_THR) {
    const int c = i & ((1 << lk) - 1), e = i >> lk, q = e / rc, b2 = e - q * rc;
    CX *p = sm + ((q * R * rc + b2) << lk) + c;
    CX v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = p[(r * rc) << lk];
    dft<R>(v, SIGN);
#pragma unroll
    for (int q2 = 0; q2 < R; q2++) {
      if (q2 > 0) {
        CX t = __ldg(tw + b2 * q2 * ra);
        if (SIGN > 0) t.y = -t.y;
        v[q2] = cmul(v[q2], t);
      }
      p[(q2 * rc) << lk] = v[q2];
    }
  }
}

// last: radix R over the values at sm[(e R + b) KXG + c], e = q rb + q2 (rb = 1 for two
// steps); store.put(v, q + ra q2, ra rb, c): output m at o + m * step
template <int R, int SIGN, typename CX, typename Store>
__device__ __forceinline__ void cols_last(CX *__restrict__ sm, int ra, int rb, int lk, Store store) {
#pragma unroll 1
  for (int i = threadIdx.x; i < (ra * rb) << lk; i += COLS_THR) {
    const int c = i & ((1 << lk) - 1), e = i >> lk;
    const int q = rb == 1 ? e : e / rb, q2 = e - q * rb;
    CX *p = sm + ((e * R) << lk) + c;
    CX v[R];
#pragma unroll
    for (int b = 0; b < R; b++) v[b] = p[b << lk];
    dft<R>(v, SIGN);
    store.template put<R>(v, q + ra * q2, ra * rb, c, p, lk);
  }
}

#define DG_COLS_RADIX(R, CALL)                       \
  switch (R) {                                       \
    case 2: { constexpr int RR = 2; CALL; } break;   \
    case 3: { constexpr int RR = 3; CALL; } break;   \
    case 4: { constexpr int RR = 4; CALL; } break;   \
    case 5: { constexpr int RR = 5; CALL; } break;   \
    case 6: { constexpr int RR = 6; CALL; } break;   \
    case 8: { constexpr int RR = 8; CALL; } break;   \
    case 9: { constexpr int RR = 9; CALL; } break;   \
    case 10: { constexpr int RR = 10; CALL; } break; \
    case 12: { constexpr int RR = 12; CALL; } break; \
    case 15: { constexpr int RR = 15; CALL; } break; \
    default: { constexpr int RR = 16; CALL; } break; \
  }

// inputs to sm up to the last step (its barrier included); NT = 0: run-time split
template <int NT, int SIGN, int LK = cols_log_kxg(NT), typename CX, typename Load>
__device__ __forceinline__ void cols_front(CX *sm, const ColPlan &pl, int lk,
                                           const CX *__restrict__ tw, Load load) {
  if constexpr (NT != 0) {
    cols_first<cols_ra(NT), SIGN>(sm, NT / cols_ra(NT), LK, tw, load);
    __syncthreads();
    if constexpr (cols_rc(NT) != 1) {
      cols_mid<cols_rb(NT), SIGN>(sm, cols_ra(NT), cols_rc(NT), LK, tw);
      __syncthreads();
    }
  } else {
    const int nb = pl.n / pl.ra;
    DG_COLS_RADIX(pl.ra, (cols_first<RR, SIGN>(sm, nb, lk, tw, load)))
    __syncthreads();
    if (pl.rc != 1) {
      DG_COLS_RADIX(pl.rb, (cols_mid<RR, SIGN>(sm, pl.ra, pl.rc, lk, tw)))
      __syncthreads();
    }
  }
}
template <int NT, int SIGN, int LK = cols_log_kxg(NT), typename CX, typename Store>
__device__ __forceinline__ void cols_back(CX *sm, const ColPlan &pl, int lk, Store store) {
  if constexpr (NT != 0) {
    constexpr int RC = cols_rc(NT);
    cols_last<RC == 1 ? cols_rb(NT) : RC, SIGN>(sm, cols_ra(NT), RC == 1 ? 1 : cols_rb(NT), LK,
                                               store);
  } else {
    const int rl = pl.rc == 1 ? pl.rb : pl.rc, rb = pl.rc == 1 ? 1 : pl.rb;
    DG_COLS_RADIX(rl, (cols_last<RR, SIGN>(sm, pl.ra, rb, lk, store)))
  }
}
#endif

}  // namespace dgfft
