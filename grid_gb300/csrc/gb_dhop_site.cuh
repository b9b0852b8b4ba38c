// gb_dhop_site.cuh -- the steps of one leg of the hopping term on a site's spinor in registers:
// projection to a two-spinor, SU(3) product, reconstruction (Grid/qcd/spin/TwoSpinor.h:75-330);
// and of the force term built on them.
#pragma once

#include "gb_device.cuh"

namespace gb {

// ---- spin projection (1 + S gamma_MU) f -> two-spinor h, Grid's spProj{X,Y,Z,T}{p,m} ----
template <int MU, int S, class R>
__device__ __forceinline__ void project(const Spinor<R>& f, R (&hr)[6], R (&hi)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const R f0r = f.re[c], f0i = f.im[c], f1r = f.re[3 + c], f1i = f.im[3 + c];
    const R f2r = f.re[6 + c], f2i = f.im[6 + c], f3r = f.re[9 + c], f3i = f.im[9 + c];
    if (MU == 0) {  // h0 = f0 + S i f3, h1 = f1 + S i f2
      hr[c] = f0r - S * f3i; hi[c] = f0i + S * f3r;
      hr[3 + c] = f1r - S * f2i; hi[3 + c] = f1i + S * f2r;
    } else if (MU == 1) {  // h0 = f0 - S f3, h1 = f1 + S f2
      hr[c] = f0r - S * f3r; hi[c] = f0i - S * f3i;
      hr[3 + c] = f1r + S * f2r; hi[3 + c] = f1i + S * f2i;
    } else if (MU == 2) {  // h0 = f0 + S i f2, h1 = f1 - S i f3
      hr[c] = f0r - S * f2i; hi[c] = f0i + S * f2r;
      hr[3 + c] = f1r + S * f3i; hi[3 + c] = f1i - S * f3r;
    } else {  // h0 = f0 + S f2, h1 = f1 + S f3
      hr[c] = f0r + S * f2r; hi[c] = f0i + S * f2i;
      hr[3 + c] = f1r + S * f3r; hi[3 + c] = f1i + S * f3i;
    }
  }
}

// ---- reconstruction, Grid's accumRecon{X,Y,Z,T}{p,m}; FIRST assigns instead of adding ----
template <int MU, int S, bool FIRST, class R>
__device__ __forceinline__ void reconstruct(Spinor<R>& r, const R (&ur)[6], const R (&ui)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const R u0r = ur[c], u0i = ui[c], u1r = ur[3 + c], u1i = ui[3 + c];
    R t2r, t2i, t3r, t3i;
    if (MU == 0) {  // r2 += -S i u1, r3 += -S i u0
      t2r = S * u1i; t2i = -S * u1r; t3r = S * u0i; t3i = -S * u0r;
    } else if (MU == 1) {  // r2 += S u1, r3 -= S u0
      t2r = S * u1r; t2i = S * u1i; t3r = -S * u0r; t3i = -S * u0i;
    } else if (MU == 2) {  // r2 += -S i u0, r3 += S i u1
      t2r = S * u0i; t2i = -S * u0r; t3r = -S * u1i; t3i = S * u1r;
    } else {  // r2 += S u0, r3 += S u1
      t2r = S * u0r; t2i = S * u0i; t3r = S * u1r; t3i = S * u1i;
    }
    if (FIRST) {
      r.re[c] = u0r; r.im[c] = u0i; r.re[3 + c] = u1r; r.im[3 + c] = u1i;
      r.re[6 + c] = t2r; r.im[6 + c] = t2i; r.re[9 + c] = t3r; r.im[9 + c] = t3i;
    } else {
      r.re[c] += u0r; r.im[c] += u0i; r.re[3 + c] += u1r; r.im[3 + c] += u1i;
      r.re[6 + c] += t2r; r.im[6 + c] += t2i; r.re[9 + c] += t3r; r.im[9 + c] += t3i;
    }
  }
}

// u = U h for both spins of the two-spinor; U is 9 complex (row-major) in shared memory
template <class R>
__device__ __forceinline__ void su3_mul(const R* __restrict__ U, const R (&hr)[6], const R (&hi)[6], R (&ur)[6],
                                        R (&ui)[6]) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const R u0r = U[(a * 3 + 0) * 2], u0i = U[(a * 3 + 0) * 2 + 1];
    const R u1r = U[(a * 3 + 1) * 2], u1i = U[(a * 3 + 1) * 2 + 1];
    const R u2r = U[(a * 3 + 2) * 2], u2i = U[(a * 3 + 2) * 2 + 1];
#pragma unroll
    for (int sp = 0; sp < 2; sp++) {
      const int o = sp * 3;
      R xr = u0r * hr[o];
      R xi = u0r * hi[o];
      xr = fma(-u0i, hi[o], xr);
      xi = fma(u0i, hr[o], xi);
      xr = fma(u1r, hr[o + 1], xr);
      xi = fma(u1r, hi[o + 1], xi);
      xr = fma(-u1i, hi[o + 1], xr);
      xi = fma(u1i, hr[o + 1], xi);
      xr = fma(u2r, hr[o + 2], xr);
      xi = fma(u2r, hi[o + 2], xi);
      xr = fma(-u2i, hi[o + 2], xr);
      xi = fma(u2i, hr[o + 2], xi);
      ur[o + a] = xr;
      ui[o + a] = xi;
    }
  }
}

// ---- force term: W += h conj(g)^T over both spins of two-spinors (W: colour c of h, b of g) ----
template <class R>
__device__ __forceinline__ void deriv_outer(const R (&hr)[6], const R (&hi)[6], const R (&gr)[6], const R (&gi)[6],
                                            double (&wr)[9], double (&wi)[9]) {
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const double xr = hr[j * 3 + c], xi = hi[j * 3 + c], yr = gr[j * 3 + b], yi = gi[j * 3 + b];
        wr[c * 3 + b] = fma(xr, yr, fma(xi, yi, wr[c * 3 + b]));
        wi[c * 3 + b] = fma(xi, yr, fma(-xr, yi, wi[c * 3 + b]));
      }
}

// The rows of U W into o (row-major 3 x 3) by the G lanes of a site that hold W: one lane all of
// them, or lane 0 rows 0, 2 and lane 1 row 1.
template <int G, class R>
__device__ __forceinline__ void deriv_rows(const R (&U)[18], const double (&wr)[9], const double (&wi)[9], int g,
                                           double2* o) {
#pragma unroll
  for (int pass = 0; pass < (G == 2 ? 2 : 3); pass++) {
    const int a = G == 2 ? (pass == 0 ? g : 2) : pass;
    if (G == 2 && pass == 1 && g == 1) break;
    double ur[3], ui[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int e = 2 * c;
      ur[c] = a == 0 ? U[e] : a == 1 ? U[6 + e] : U[12 + e];
      ui[c] = a == 0 ? U[e + 1] : a == 1 ? U[7 + e] : U[13 + e];
    }
#pragma unroll
    for (int b = 0; b < 3; b++) {
      double re = 0, im = 0;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        re = fma(ur[c], wr[c * 3 + b], fma(-ui[c], wi[c * 3 + b], re));
        im = fma(ur[c], wi[c * 3 + b], fma(ui[c], wr[c * 3 + b], im));
      }
      o[a * 3 + b] = make_double2(re, im);
    }
  }
}

// the lexicographic site of x_cb on checkerboard `parity`
__device__ __forceinline__ int64_t site_of_cb(const int (&L)[4], int parity, int64_t x) {
  const int Lxh = L[0] >> 1;
  const int64_t row = x / Lxh;
  const int xh = int(x - row * Lxh);
  const int y = int(row % L[1]);
  const int64_t zt = row / L[1];
  const int z = int(zt % L[2]), t = int(zt / L[2]);
  return row * L[0] + 2 * xh + ((parity + y + z + t) & 1);
}

}  // namespace gb
