// Column transforms of the substeps (fft_cols.cuh): spectral planes to
// half-physical planes and back, and the channel's z forward that writes the
// nonlinear term.
#include "dg_internal.cuh"
#include "fft_cols.cuh"

using namespace dgfft;

namespace {

// bins k = b + nb r of columns c0 .. of a packed spectral plane, zero in the
// truncated band (NK, N - NK)
template <typename CI, typename CX>
struct LoadModes {
  const CI *in;  // the plane's column c0
  int n, nk, rowlen, ncol;
  template <int R>
  __device__ __forceinline__ void get(CX *v, int b, int nb, int c) const {
    using T = typename CT<CX>::T;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int z = b + nb * r;
      const int kp = z <= nk ? z : z - n + 1 + 2 * nk;
      CI x{};
      if (c < ncol && (z <= nk || z >= n - nk)) x = in[(long)kp * rowlen + c];
      v[r] = CT<CX>::mk((T)x.x, (T)x.y);
    }
  }
};

template <typename CX>
struct LoadBins {
  const CX *in;
  int rowlen, ncol;
  template <int R>
  __device__ __forceinline__ void get(CX *v, int b, int nb, int c) const {
#pragma unroll
    for (int r = 0; r < R; r++)
      v[r] = c < ncol ? in[(long)(b + nb * r) * rowlen + c] : CT<CX>::mk(0, 0);
  }
};

// PK, and pk given: *pk becomes the largest component's magnitude of the columns but cskip
template <typename CX, bool PK>
struct StoreBins {
  CX *out;
  int rowlen, ncol;
  unsigned *pk;
  int cskip;
  template <int R>
  __device__ __forceinline__ void put(CX *v, int o, int step, int c, CX *, int) const {
    if (c >= ncol) return;
#pragma unroll
    for (int m = 0; m < R; m++) out[(long)(o + m * step) * rowlen + c] = v[m];
    if (PK && pk) {
      unsigned t = 0;
#pragma unroll
      for (int m = 0; m < R; m++) t = max(t, max(dg_mag(v[m].x), dg_mag(v[m].y)));
      if (c != cskip) *pk = max(*pk, t);
    }
  }
};

// retained bins, scaled by 1/N, to packed slots
template <typename CX, typename CO>
struct StoreModes {
  CO *out;
  int n, nk, rowlen, ncol;
  double rn;
  template <int R>
  __device__ __forceinline__ void put(CX *v, int o, int step, int c, CX *, int) const {
    using T = typename CT<CO>::T;
    if (c >= ncol) return;
#pragma unroll
    for (int m = 0; m < R; m++) {
      const int z = o + m * step;
      if (z > nk && z < n - nk) continue;
      const int kp = z <= nk ? z : z - n + 1 + 2 * nk;
      out[(long)kp * rowlen + c] =
          CT<CO>::mk((T)((double)v[m].x * rn), (T)((double)v[m].y * rn));
    }
  }
};

template <int NT, bool PK, typename CI, typename CX>
__global__ void __launch_bounds__(COLS_THR, 4)
    k_cols_inv(PtrArray<const CI> fields, int jmin, long in_plane, int rowlen, int nk, ColPlan pl,
               int lk, const CX *__restrict__ tw, CX *__restrict__ H, long out_field, PeakOut peak) {
  extern __shared__ double2 sm_raw[];
  CX *sm = reinterpret_cast<CX *>(sm_raw);
  const int n = NT ? NT : pl.n, kxg = 1 << (NT ? cols_log_kxg(NT) : lk);
  const int c0 = blockIdx.x * kxg, j = jmin + blockIdx.y, f = blockIdx.z;
  const int ncol = min(kxg, rowlen - c0);
  dg_pdl_wait();
  cols_front<NT, +1>(sm, pl, lk, tw,
                     LoadModes<CI, CX>{fields(f) + (long)j * in_plane + c0, n, nk, rowlen, ncol});
  unsigned pk = 0;
  const bool want = PK && (f == 0 || f >= 3);  // U1 and the scalars
  cols_back<NT, +1>(sm, pl, lk,
                    StoreBins<CX, PK>{H + f * out_field + (long)j * n * rowlen + c0, rowlen, ncol,
                                      want ? &pk : nullptr, peak.skip0 && c0 == 0 ? 0 : -1});
  if (PK && want) {
    pk = __reduce_max_sync(0xffffffffu, pk);
    if ((threadIdx.x & 31) == 0)
      peak.p[(((long)f * peak.planes + j) * gridDim.x + blockIdx.x) * (COLS_THR / 32) +
             (threadIdx.x >> 5)] = pk;
  }
}

template <int NT, typename CX, typename CO>
__global__ void __launch_bounds__(COLS_THR, 4)
    k_cols_fwd(const CX *__restrict__ H, long in_field, int jmin, int rowlen, int nk, ColPlan pl,
               int lk, const CX *__restrict__ tw, PtrArray<CO> fields, long out_plane) {
  extern __shared__ double2 sm_raw[];
  CX *sm = reinterpret_cast<CX *>(sm_raw);
  const int n = NT ? NT : pl.n, kxg = 1 << (NT ? cols_log_kxg(NT) : lk);
  const int c0 = blockIdx.x * kxg, j = jmin + blockIdx.y, f = blockIdx.z;
  const int ncol = min(kxg, rowlen - c0);
  dg_pdl_wait();
  cols_front<NT, -1>(sm, pl, lk, tw,
                     LoadBins<CX>{H + f * in_field + (long)j * n * rowlen + c0, rowlen, ncol});
  cols_back<NT, -1>(sm, pl, lk,
                    StoreModes<CX, CO>{fields(f) + (long)j * out_plane + c0, n, nk, rowlen, ncol,
                                       1.0 / (double)n});
}

// The channel's z forward: both product arrays of a field, A and B, on one
// plane, and the nonlinear term -i kz A + B of every retained mode.  A goes
// first; its outputs stay in the slots of shared memory they came from until
// B's are there (StoreNl takes them times -i kz).
template <typename CX>
struct KeepA {
  template <int R>
  __device__ __forceinline__ void put(CX *v, int o, int step, int, CX *p, int lk) const {
#pragma unroll
    for (int m = 0; m < R; m++) p[m << lk] = v[m];
  }
};
template <typename CX>
struct StoreNl {
  double2 *out;
  const CX *a;     // A's outputs, in the layout of sm
  const CX *smb;   // B's buffer: the same slots
  const double *kz;
  int n, nk, rowlen, ncol;
  double rn;
  template <int R>
  __device__ __forceinline__ void put(CX *v, int o, int step, int c, CX *p, int lk) const {
    if (c >= ncol) return;
    const CX *pa = a + (p - smb);
#pragma unroll
    for (int m = 0; m < R; m++) {
      const int z = o + m * step;
      if (z > nk && z < n - nk) continue;
      const int kp = z <= nk ? z : z - n + 1 + 2 * nk;
      const CX aw = pa[m << lk];
      const double K = __ldg(kz + kp);
      out[(long)kp * rowlen + c] = make_double2(K * ((double)aw.y * rn) + (double)v[m].x * rn,
                                                -K * ((double)aw.x * rn) + (double)v[m].y * rn);
    }
  }
};

struct NlRows {
  int lo[3 + DG_MAX_TH], hi[3 + DG_MAX_TH];
};

// Two buffers: half the columns per CTA above 256 points, for four CTAs per SM
// (64x65x512 with a scalar: 84 -> 59 us).
__host__ __device__ constexpr int nl_log_kxg(int n) {
  return n > 256 && n <= 512 ? 2 : cols_log_kxg(n);
}

template <int NT, typename CX>
__global__ void __launch_bounds__(COLS_THR, 4)
    k_cols_nl(const CX *__restrict__ G, long gfield, int jmin, int rowlen, int nk, ColPlan pl,
              int lk, const CX *__restrict__ tw, const double *__restrict__ kz, FieldPtrs rhs,
              long out_plane, NlRows rows) {
  extern __shared__ double2 sm_raw[];
  constexpr int LK = nl_log_kxg(NT);
  const int n = NT ? NT : pl.n, kxg = 1 << (NT ? LK : lk);
  CX *sa = reinterpret_cast<CX *>(sm_raw), *sb = sa + n * kxg;
  const int c0 = blockIdx.x * kxg, j = jmin + blockIdx.y, f = blockIdx.z;
  int lo = rows.lo[0], hi = rows.hi[0];
#pragma unroll
  for (int q = 1; q < 3 + DG_MAX_TH; q++) {
    lo = f == q ? rows.lo[q] : lo;
    hi = f == q ? rows.hi[q] : hi;
  }
  if (j < lo || j > hi) return;
  const int ncol = min(kxg, rowlen - c0);
  dg_pdl_wait();  // G comes from the x-row kernel
  const CX *ga = G + (2 * f) * gfield + (long)j * n * rowlen + c0;
  const double rn = 1.0 / (double)n;
  cols_front<NT, -1, LK>(sa, pl, lk, tw, LoadBins<CX>{ga, rowlen, ncol});
  cols_front<NT, -1, LK>(sb, pl, lk, tw, LoadBins<CX>{ga + gfield, rowlen, ncol});
  // each thread keeps A's outputs in the slots it reads them from, and takes
  // the same items again for B: no barrier between
  cols_back<NT, -1, LK>(sa, pl, lk, KeepA<CX>{});
  cols_back<NT, -1, LK>(sb, pl, lk,
                    StoreNl<CX>{rhs(f) + (long)j * out_plane + c0, sa, sb, kz, n, nk, rowlen, ncol,
                                rn});
}

// the split and the launch shape of length n; false where there is none
template <typename CX>
bool cols_shape(int n, ColPlan *pl, int *lk, size_t *sm) {
  if (cols_ra(n)) *pl = {n, cols_ra(n), cols_rb(n), cols_rc(n)};
  else if (!cols_plan(n, pl)) return false;
  *lk = cols_log_kxg(n);
  *sm = (sizeof(CX) * (size_t)n) << *lk;
  return true;
}

template <typename CI, typename CX>
int inv_t(dg_handle *h, const CI *const *fields, int nf, int jmin, int jmax, long in_plane,
          int rowlen, int n, int nk, const CX *tw, CX *H, long out_field, PeakOut peak,
          const char *name) {
  ColPlan pl;
  int lk;
  size_t sm;
  if (!cols_shape<CX>(n, &pl, &lk, &sm)) return 1;
  if (jmax < jmin || nf <= 0) return DG_OK;
  PtrArray<const CI> fp{};
  for (int f = 0; f < nf; f++) fp.p[f] = fields[f];
  const dim3 grid(dg_cdiv(rowlen, 1 << lk), jmax - jmin + 1, nf);
#define KERNEL_BODY(NN)                                                                        \
  {                                                                                            \
    auto kern = peak.p ? k_cols_inv<NN, true, CI, CX> : k_cols_inv<NN, false, CI, CX>;         \
    dg_big_smem((const void *)kern);                                                           \
    dg_kt_begin(h, name, h->st);                                                               \
    DG_CUDA(dg_launch(h->pdl_zinv, kern, grid, dim3(COLS_THR), sm, h->st, fp, jmin, in_plane,  \
                      rowlen, nk, pl, lk, tw, H, out_field, peak));                            \
  }
  switch (n) {
    DG_FOR_EACH_N(DG_CASE_N)
    default: KERNEL_BODY(0); break;
  }
#undef KERNEL_BODY
  DG_LAUNCHED();
  return DG_OK;
}

template <typename CX, typename CO>
int fwd_t(dg_handle *h, const CX *H, long in_field, int nf, int jmin, int jmax, int rowlen, int n,
          int nk, const CX *tw, CO *const *fields, long out_plane, const char *name) {
  ColPlan pl;
  int lk;
  size_t sm;
  if (!cols_shape<CX>(n, &pl, &lk, &sm)) return 1;
  if (jmax < jmin || nf <= 0) return DG_OK;
  PtrArray<CO> fp{};
  for (int f = 0; f < nf; f++) fp.p[f] = fields[f];
  const dim3 grid(dg_cdiv(rowlen, 1 << lk), jmax - jmin + 1, nf);
#define KERNEL_BODY(NN)                                                                        \
  {                                                                                            \
    auto kern = k_cols_fwd<NN, CX, CO>;                                                        \
    dg_big_smem((const void *)kern);                                                           \
    dg_kt_begin(h, name, h->st);                                                               \
    DG_CUDA(dg_launch(0, kern, grid, dim3(COLS_THR), sm, h->st, H, in_field, jmin, rowlen, nk, \
                      pl, lk, tw, fp, out_plane));                                             \
  }
  switch (n) {
    DG_FOR_EACH_N(DG_CASE_N)
    default: KERNEL_BODY(0); break;
  }
#undef KERNEL_BODY
  DG_LAUNCHED();
  return DG_OK;
}

template <typename CX>
int nl_t(dg_handle *h, const CX *G, const CX *tw, int jmin, int jmax, const char *name) {
  ColPlan pl;
  int lk;
  size_t sm;
  if (!cols_shape<CX>(h->NZ, &pl, &lk, &sm)) return 1;
  lk = nl_log_kxg(h->NZ);
  sm = (sizeof(CX) * (size_t)h->NZ) << lk;
  if (2 * sm > 220 * 1024) return 1;
  if (jmax < jmin) return DG_OK;
  FieldPtrs rhs{};
  NlRows rows{};
  for (int f = 0; f < h->nf; f++) {
    rhs.p[f] = h->rhs[f];
    rows.lo[f] = f == 1 ? 2 : f < 3 ? h->jstart : h->jstart_th[f - 3];
    rows.hi[f] = f == 1 ? h->NY : f < 3 ? h->jend : h->jend_th[f - 3];
  }
  const long gfield = (long)h->nplanes * h->NZ * h->nkxp;
  const dim3 grid(dg_cdiv(h->nkxp, 1 << lk), jmax - jmin + 1, h->nf);
#define KERNEL_BODY(NN)                                                                         \
  {                                                                                             \
    auto kern = k_cols_nl<NN, CX>;                                                              \
    dg_big_smem((const void *)kern);                                                            \
    dg_kt_begin(h, name, h->st);                                                                \
    DG_CUDA(dg_launch(h->pdl, kern, grid, dim3(COLS_THR), 2 * sm, h->st, G, gfield, jmin,       \
                      h->nkxp, h->NKZ, pl, lk, tw, h->kz, rhs, h->ss, rows));                   \
  }
  switch (h->NZ) {
    DG_FOR_EACH_N(DG_CASE_N)
    default: KERNEL_BODY(0); break;
  }
#undef KERNEL_BODY
  DG_LAUNCHED();
  return DG_OK;
}

}  // namespace

int dg_cols_group(int n) {
  ColPlan pl;
  return cols_ra(n) || cols_plan(n, &pl) ? 1 << cols_log_kxg(n) : 0;
}

int dg_cols_inv(dg_handle *h, const double2 *const *f, int nf, int jmin, int jmax, long in_plane,
                int rowlen, int n, int nk, const double2 *tw, double2 *H, long out_field,
                PeakOut peak) {
  return inv_t(h, f, nf, jmin, jmax, in_plane, rowlen, n, nk, tw, H, out_field, peak, "k_cols_inv");
}
int dg_cols_inv(dg_handle *h, const double2 *const *f, int nf, int jmin, int jmax, long in_plane,
                int rowlen, int n, int nk, const float2 *tw, float2 *H, long out_field,
                PeakOut peak) {
  return inv_t(h, f, nf, jmin, jmax, in_plane, rowlen, n, nk, tw, H, out_field, peak, "k_cols_inv_f32");
}
int dg_cols_inv(dg_handle *h, const float2 *const *f, int nf, int jmin, int jmax, long in_plane,
                int rowlen, int n, int nk, const float2 *tw, float2 *H, long out_field,
                PeakOut peak) {
  return inv_t(h, f, nf, jmin, jmax, in_plane, rowlen, n, nk, tw, H, out_field, peak, "k_cols_inv_f32");
}
int dg_cols_fwd(dg_handle *h, const double2 *H, long in_field, int nf, int jmin, int jmax,
                int rowlen, int n, int nk, const double2 *tw, double2 *const *f, long out_plane) {
  return fwd_t(h, H, in_field, nf, jmin, jmax, rowlen, n, nk, tw, f, out_plane, "k_cols_fwd");
}
int dg_cols_fwd(dg_handle *h, const float2 *H, long in_field, int nf, int jmin, int jmax,
                int rowlen, int n, int nk, const float2 *tw, float2 *const *f, long out_plane) {
  return fwd_t(h, H, in_field, nf, jmin, jmax, rowlen, n, nk, tw, f, out_plane, "k_cols_fwd_f32");
}
int dg_cols_nl(dg_handle *h, int jmin, int jmax) {
  if (h->mixed)
    return nl_t<float2>(h, reinterpret_cast<const float2 *>(h->G), h->twz_f, jmin, jmax,
                        "k_cols_nl_f32");
  return nl_t<double2>(h, h->G, h->twz, jmin, jmax, "k_cols_nl");
}
