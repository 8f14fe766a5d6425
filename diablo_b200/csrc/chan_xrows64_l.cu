// k_xrows (chan_xrows.cuh) for 72 to 160 points, FP64.
#include "chan_xrows.cuh"

int dg_xrows64_l(dg_handle *h, int ja, int jb);

int dg_xrows64_l(dg_handle *h, int ja, int jb) {
  const double2 *H = h->H, *tw = h->twx;
  switch (h->NX) {
    case 72: return xr_th<9, 8, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 80: return xr_th<16, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 90: return xr_th<15, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 120: return xr_th<15, 8, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 160: return xr_th<32, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    default: return DG_ERR_ARG;
  }
}
