// k_xrows (chan_xrows.cuh) for the lengths 2^a 3^b that both precisions take.
#include "chan_xrows.cuh"

namespace {

template <typename CX>
int xr_dispatch(dg_handle *h, int ja, int jb, const CX *H, const CX *tw, CX *G, const char *name) {
  switch (h->NX) {
    case 16: return xr_th<4, 4, CX>(h, ja, jb, H, tw, G, name);
    case 32: return xr_th<8, 4, CX>(h, ja, jb, H, tw, G, name);
    case 48: return xr_th<8, 6, CX>(h, ja, jb, H, tw, G, name);
    case 64: return xr_th<8, 8, CX>(h, ja, jb, H, tw, G, name);
    case 96: return xr_th<16, 6, CX>(h, ja, jb, H, tw, G, name);
    default: return xr_th<16, 8, CX>(h, ja, jb, H, tw, G, name);
  }
}

}  // namespace

bool dg_xrows_ok(const dg_handle *h) {
  const int n = h->NX;
  const bool both = n == 16 || n == 32 || n == 48 || n == 64 || n == 96 || n == 128;
  return h->NTH <= 2 && (both || (!h->mixed && dg_xrows64_ok(n, h->NTH)));
}

// output planes ja..jb (H holds ja-1..jb+1)
int dg_xrows(dg_handle *h, int ja, int jb) {
  if (h->mixed)
    return xr_dispatch(h, ja, jb, reinterpret_cast<const float2 *>(h->H), (const float2 *)h->twx_f,
                       reinterpret_cast<float2 *>(h->G), "k_xrows_f32");
  if (dg_xrows64_ok(h->NX, h->NTH)) return dg_xrows64(h, ja, jb);
  return xr_dispatch(h, ja, jb, (const double2 *)h->H, (const double2 *)h->twx, h->G, "k_xrows");
}
