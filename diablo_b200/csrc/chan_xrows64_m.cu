// k_xrows (chan_xrows.cuh) for 50 to 180 points, FP64.
#include "chan_xrows.cuh"

int dg_xrows64_m(dg_handle *h, int ja, int jb);

int dg_xrows64_m(dg_handle *h, int ja, int jb) {
  const double2 *H = h->H, *tw = h->twx;
  switch (h->NX) {
    case 50: return xr_th<10, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 100: return xr_th<20, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 108: return xr_th<18, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 144: return xr_th<24, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 150: return xr_th<30, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 162: return xr_th<18, 9, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 180: return xr_th<30, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    default: return DG_ERR_ARG;
  }
}
