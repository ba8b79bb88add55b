// FP64 pair terms on the device that are cheaper than the bit-identical ones of
// wn_pair.cuh where those bits cannot matter.
#pragma once

#include "wn_common.cuh"
#include "wn_pair.cuh"

namespace wn {

// det and denom of a pair (wn_pair.cuh) with contracted products and rsqrt64's roots: 65
// FP64 operations instead of 115. True if denom is certain to be positive by a margin
// (above |a||b||c| / 4, and between 2^-300 and 2^300): then no branch of the angle is
// near, its error stays within a few roundings, and neither term's last bits decide
// anything. Else, and for anything not finite, the caller takes the bit-identical terms.
__device__ __forceinline__ bool pair_terms_far(double ox, double oy, double oz, double Ax,
                                               double Ay, double Az, double Bx, double By,
                                               double Bz, double Cx, double Cy, double Cz,
                                               double& det, double& denom) {
  const double ax = Ax - ox, ay = Ay - oy, az = Az - oz;
  const double bx = Bx - ox, by = By - oy, bz = Bz - oz;
  const double cx = Cx - ox, cy = Cy - oy, cz = Cz - oz;
  const double aa = fma(ax, ax, fma(ay, ay, az * az));
  const double bb = fma(bx, bx, fma(by, by, bz * bz));
  const double cc = fma(cx, cx, fma(cy, cy, cz * cz));
  const double la = aa * rsqrt64(aa), lb = bb * rsqrt64(bb), lc = cc * rsqrt64(cc);
  const double nx = fma(by, cz, -(bz * cy)), ny = fma(bz, cx, -(bx * cz)),
               nz = fma(bx, cy, -(by * cx));
  det = fma(ax, nx, fma(ay, ny, az * nz));
  const double lll = la * lb * lc;
  double d = fma(fma(ax, bx, fma(ay, by, az * bz)), lc, lll);
  d = fma(fma(bx, cx, fma(by, cy, bz * cz)), la, d);
  denom = fma(fma(cx, ax, fma(cy, ay, cz * az)), lb, d);
  const int hd = __double2hiint(denom);  // high words order positive numbers
  return hd > 0x2d300000 && hd < 0x52b00000 && hd > __double2hiint(lll) - 0x00200000;
}

// Adds two faces to a query's product. Both factors far: their arguments lie within
// (-pi/2, pi/2), so they multiply without a turn and go in as one.
__device__ __forceinline__ void push_two(ArgAcc& acc, double ox, double oy, double oz,
                                         const double (&u)[9], const double (&v)[9]) {
  double t0, d0, t1, d1;
  const bool far0 = pair_terms_far(ox, oy, oz, u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7],
                                   u[8], t0, d0);
  const bool far1 = pair_terms_far(ox, oy, oz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7],
                                   v[8], t1, d1);
  if (far0 && far1) {
    argacc_push(acc, fma(d0, d1, -(t0 * t1)), fma(d0, t1, t0 * d1));
    return;
  }
  if (!far0)
    pair_terms_exact(ox, oy, oz, u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], u[8], t0, d0);
  argacc_push(acc, d0, t0);
  if (!far1)
    pair_terms_exact(ox, oy, oz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], t1, d1);
  argacc_push(acc, d1, t1);
}

__device__ __forceinline__ void push_one(ArgAcc& acc, double ox, double oy, double oz,
                                         const double (&v)[9]) {
  double t, d;
  if (!pair_terms_far(ox, oy, oz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], t, d))
    pair_terms_exact(ox, oy, oz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], t, d);
  argacc_push(acc, d, t);
}

}  // namespace wn
