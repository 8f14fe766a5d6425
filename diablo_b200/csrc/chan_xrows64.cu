// k_xrows (chan_xrows.cuh) in FP64 for further lengths with factors 2, 3 and 5: the
// rule, the dispatch and the shortest ones.  They replaced a c2r launch and a
// launch per product pair with run-time transform plans (per launch, a scalar: 60x33x30 30 -> 16 us,
// 150x65x48 101 -> 34, 72x74x324 261 -> 76, 240x65x48 147 -> 53; 320x65x48 with two 196 -> 132).
#include "chan_xrows.cuh"

int dg_xrows64_l(dg_handle *h, int ja, int jb);
int dg_xrows64_m(dg_handle *h, int ja, int jb);
int dg_xrows64_x(dg_handle *h, int ja, int jb);

// Rows of 256 points with scalars stay with k_xmarch: the points of four and
// more fields (8 per lane) spill here (256x129x64 with a scalar: 126 us against 117;
// without, 256x65x32: 27 against 33).
bool dg_xrows64_ok(int n, int nth) {
  switch (n) {
    case 20: case 24: case 30: case 36: case 40: case 50: case 54: case 60: case 72: case 80:
    case 90: case 100: case 108: case 120: case 144: case 150: case 160: case 162: case 180:
    case 192: case 216: case 240: case 270: case 288: case 320: return true;
    case 256: return nth == 0;
    default: return false;
  }
}

int dg_xrows64(dg_handle *h, int ja, int jb) {
  const double2 *H = h->H, *tw = h->twx;
  switch (h->NX) {
    case 20: return xr_th<5, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 24: return xr_th<6, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 30: return xr_th<6, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 36: return xr_th<9, 4, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 40: return xr_th<8, 5, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 54: return xr_th<9, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 60: return xr_th<10, 6, double2>(h, ja, jb, H, tw, h->G, "k_xrows");
    case 72: case 80: case 90: case 120: case 160: return dg_xrows64_l(h, ja, jb);
    case 192: case 216: case 240: case 256: case 270: case 288: case 320: return dg_xrows64_x(h, ja, jb);
    default: return dg_xrows64_m(h, ja, jb);
  }
}
