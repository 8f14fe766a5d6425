// k_xrows (chan_xrows.cuh) for lengths with a factor 5 or 9, FP64: the shorter ones,
// and the dispatch.
#include "chan_xrows.cuh"

int dg_xrows5_long(dg_handle *h, int ja, int jb);

bool dg_xrows5_ok(int n) {
  switch (n) {
    case 20:
    case 24:
    case 30:
    case 36:
    case 40:
    case 54:
    case 60:
    case 72:
    case 80:
    case 90:
    case 120:
    case 160:
      return true;
    default: return false;
  }
}

int dg_xrows5(dg_handle *h, int ja, int jb) {
  const double2 *H = h->H, *tw = h->twx;
  switch (h->NX) {
    case 20: return xr_th<5, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 24: return xr_th<6, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 30: return xr_th<6, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 36: return xr_th<9, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 40: return xr_th<8, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 54: return xr_th<9, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 60: return xr_th<10, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    default: return dg_xrows5_long(h, ja, jb);
  }
}
