// Fields of a straight segment carrying a constant displacement discontinuity
// (the 2DS0 element: plane strain, full space), host and device.
//
// Published solution: Crouch & Starfield, "Boundary Element Methods in Solid
// Mechanics" (1983), section 5.2.  For a segment |x| <= a on y = 0 with DD
// (Dx, Dy) (shear, normal) and
//   f(x, y) = -c [ y (atan2(y, x - a) - atan2(y, x + a))
//                  - (x - a) ln r1 + (x + a) ln r2 ],   c = 1 / (4 pi (1 - nu)),
// r1^2 = (x - a)^2 + y^2, r2^2 = (x + a)^2 + y^2, the displacements and stresses
// are linear in the derivatives of f:
//   ux  = Dx [2(1 - nu) f_y - y f_xx] + Dy [-(1 - 2nu) f_x - y f_xy]
//   uy  = Dx [(1 - 2nu) f_x - y f_xy] + Dy [2(1 - nu) f_y - y f_yy]
//   sxx = 2G Dx [2 f_xy + y f_xyy] + 2G Dy [f_yy + y f_yyy]
//   syy = 2G Dx [-y f_xyy]         + 2G Dy [f_yy - y f_yyy]
//   sxy = 2G Dx [f_yy + y f_yyy]   + 2G Dy [-y f_xyy]
// This is the element of the reference's 2DS0-H kernel (its own closed forms
// are written for the unit segment: We_segment_0 / Se_segment_0,
// src/elasticity/fullspace_iso_2d_segment/elastic_2dP0_segment.cc:82-211); the
// stresses agree with its observation kernel W (bie_elastostatic_segment_0_
// influence.h:320-372).  On the element's own line (y = 0, |x| < a) the
// displacement jumps; like the reference, y = 0 is taken as the limit from
// below (y -> 0-).
//
// Frames (src/elements/segment.h:40-90): t = (v1 - v0) / |v1 - v0|, n = (-t_y,
// t_x); local = R global with R's rows t, n; a stress tensor maps back as
// R^T S R and a vector as R^T u.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define BW_S0_HD __host__ __device__ __forceinline__
#else
#define BW_S0_HD inline
#endif

namespace bw {
namespace s0 {

// One element: centre, half length, unit tangent.
constexpr int kRecordDoubles = 5;  // cx, cy, a, tx, ty
constexpr double kPi = 3.14159265358979323846;

// Derivatives of F = f / c (f_xx = -f_yy).  With z = x + i y, both end points
// combine into one complex reciprocal,
//   1 / (z - a) - 1 / (z + a) = 2 a / zeta,          zeta = z^2 - a^2,
//   1 / (z - a)^2 - 1 / (z + a)^2 = 4 a z / zeta^2,
// |zeta|^2 = r1^2 r2^2, whose parts are the second and third derivatives; the
// two logarithms are one of the ratio and the two angles one, the angle the
// segment subtends.  A pair costs one division, one log and one atan2 (eight
// divisions and two of each when every term is taken by itself), and the
// derivatives lose no digits to the difference of two nearly equal ends in the
// far field.  f_x does: the logarithm of a ratio near 1 has an error of eps x
// distance / length (3e-15 at 100 half lengths, a tenth of the term-by-term
// form's).
struct Derivs {
  double fx, fy, fxy, fyy, fxyy, fyyy;
};

BW_S0_HD Derivs derivs(double x, double y, double a) {
  const double xm = x - a, xp = x + a, y2 = y * y;
  const double r1 = xm * xm + y2, r2 = xp * xp + y2;  // squared distances to the ends
  const double w = 1.0 / (r1 * r2);
  const double zr = xm * xp - y2, zi = 2.0 * x * y;   // zeta, no cancellation near an end
  const double gr = zr * w, gi = -zi * w;             // 1 / zeta
  const double hr = gr * gr - gi * gi, hi = 2.0 * gr * gi;
  const double ys = (y == 0.0) ? -0.0 : y;            // on the line: the limit from below
  Derivs d;
  d.fx = 0.5 * log(r1 * r1 * w);
  d.fy = -atan2(2.0 * a * ys, xm * xp + y2);
  d.fyy = -2.0 * a * gr;
  d.fxy = -2.0 * a * gi;
  d.fxyy = 4.0 * a * (x * hr - y * hi);
  d.fyyy = -4.0 * a * (x * hi + y * hr);
  return d;
}

// What a field evaluation reads of an element: centre, half length, tangent,
// cosine and sine of its double angle, the local DD over 4 pi (1 - nu).
constexpr int kFieldDoubles = 9;

BW_S0_HD void field_data(const double *rec, double dd_s, double dd_n, double nu, double *el) {
  const double tx = rec[3], ty = rec[4], c = 1.0 / (4.0 * kPi * (1.0 - nu));
  for (int k = 0; k < 5; k++) el[k] = rec[k];
  el[5] = tx * tx - ty * ty;
  el[6] = 2.0 * tx * ty;
  el[7] = c * dd_s;
  el[8] = c * dd_n;
}

// Global stress (s11, s22, s12) and displacement (u1, u2) at point (px, py)
// due to the element `el` (field_data), added to acc (5 values: s11, s22, s12,
// u1, u2).  The local stress enters through its mean m, half difference h and
// shear q, which rotate by the double angle.
template <bool kStress, bool kDisp>
BW_S0_HD void add_fields(const double *el, double px, double py, double G, double nu, double acc[5]) {
  const double tx = el[3], ty = el[4], us = el[7], un = el[8];
  const double dx = px - el[0], dy = py - el[1];
  const double x = tx * dx + ty * dy, y = tx * dy - ty * dx;
  const Derivs d = derivs(x, y, el[2]);
  if (kStress) {
    const double ks = 2.0 * G * us, kn = 2.0 * G * un;
    const double p = y * d.fxyy, r = y * d.fyyy;
    // sxx = ks (2 fxy + p) + kn (fyy + r), syy = -ks p + kn (fyy - r), sxy = ks (fyy + r) - kn p
    const double m = ks * d.fxy + kn * d.fyy, h = ks * (d.fxy + p) + kn * r, q = ks * (d.fyy + r) - kn * p;
    const double v = h * el[5] - q * el[6];
    acc[0] += m + v;
    acc[1] += m - v;
    acc[2] += h * el[6] + q * el[5];
  }
  if (kDisp) {
    const double k1 = 2.0 * (1.0 - nu), k2 = 1.0 - 2.0 * nu;
    const double ux = us * (k1 * d.fy + y * d.fyy) - un * (k2 * d.fx + y * d.fxy);
    const double uy = us * (k2 * d.fx - y * d.fxy) + un * (k1 * d.fy - y * d.fyy);
    acc[3] += ux * tx - uy * ty;
    acc[4] += ux * ty + uy * tx;
  }
}

// The same from the element's record and its local DD (dd_s, dd_n).
template <bool kStress = true, bool kDisp = true>
BW_S0_HD void add_point_fields(const double *rec, double dd_s, double dd_n, double px, double py, double G,
                               double nu, double acc[5]) {
  double el[kFieldDoubles];
  field_data(rec, dd_s, dd_n, nu, el);
  add_fields<kStress, kDisp>(el, px, py, G, nu, acc);
}

// Hypersingular (H) entry between two elements: tractions at the receiver's
// centre, in the receiver's frame (shear along its tangent, normal along its
// normal), due to unit local DDs of the source; K[j][k] = traction j due to
// DD k.  The reference's BieElastostatic<Segment<0>, Segment<0>, H>
// (bie_elastostatic_segment_0_influence.h:176-232) stores the same 2 x 2
// block column-major.
BW_S0_HD void h_entry(const double *src, const double *rcv, double G, double nu, double K[2][2]) {
  const double tx = rcv[3], ty = rcv[4], nx = -ty, ny = tx;
  for (int k = 0; k < 2; k++) {
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    add_point_fields<true, false>(src, k == 0 ? 1.0 : 0.0, k == 1 ? 1.0 : 0.0, rcv[0], rcv[1], G, nu, acc);
    const double t1 = acc[0] * nx + acc[2] * ny, t2 = acc[2] * nx + acc[1] * ny;  // sigma n
    K[0][k] = t1 * tx + t2 * ty;
    K[1][k] = t1 * nx + t2 * ny;
  }
}

}  // namespace s0
}  // namespace bw
