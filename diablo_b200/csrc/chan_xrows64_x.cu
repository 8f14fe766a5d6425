// k_xrows (chan_xrows.cuh) for 192 to 320 points, FP64.
#include "chan_xrows.cuh"

int dg_xrows64_x(dg_handle *h, int ja, int jb);

int dg_xrows64_x(dg_handle *h, int ja, int jb) {
  const double2 *H = h->H, *tw = h->twx;
  switch (h->NX) {
    case 192: return xr_th<24, 8, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 256: return xr_launch<32, 8, 0, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 320: return xr_th<32, 10, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 216: return xr_th<24, 9, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 240: return xr_th<30, 8, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 270: return xr_th<30, 9, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 288: return xr_th<32, 9, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    default: return DG_ERR_ARG;
  }
}
