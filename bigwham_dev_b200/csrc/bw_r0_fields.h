// Fields at a point due to a rectangular element carrying a constant
// displacement discontinuity (3DR0), in the global frame, host and device:
// the element's local stresses and displacements (bw_r0.h: the reference's
// StressesKernelR0 / DisplacementKernelR0 restated) contracted with the local
// DD and rotated back, sigma_g = R^T sigma_l R, u_g = R^T u_l (R row-major,
// local = R global).  The reference's BigWhamIO has no working 3DR0
// observation kernel (BieElastostatic<Rectangle<0>, Point<3>, T | W> return
// zeros, bie_elastostatic_rectangle_0_influence.h:222-245); the output
// layout is the one its 3D observation kernels use
// (bie_elastostatic_triangle_0_influence.h:196-215): s11, s22, s33, s12,
// s13, s23 and u1, u2, u3.
#pragma once

#include "bw_r0.h"

namespace bw {
namespace r0 {

// Element data a field evaluation reads: collocation point (3), rotation
// row-major (9), half sides a, b; then the local DD (3).
constexpr int kFieldDoubles = 17;

// el: kFieldDoubles values as above; acc += the 9 field values at p.  The DD
// contracts with the derivatives directly (bw_r0.h's table of stresses and
// displacements, with the coefficients of each derivative collected).
template <bool kStress = true, bool kDisp = true>
BW_HD void add_point_fields(const double *el, const double *p, double G, double nu, double acc[9]) {
  const double *cp = el, *R = el + 3, *dd = el + 14;
  const double a = el[12], b = el[13];
  double d[3], l[3];
  for (int k = 0; k < 3; k++) d[k] = p[k] - cp[k];
  for (int i = 0; i < 3; i++) l[i] = R[3 * i] * d[0] + R[3 * i + 1] * d[1] + R[3 * i + 2] * d[2];
  const Derivs D = derivs(l[0], l[1], l[2], a, b);
  const double z = l[2], k2 = 1.0 - 2.0 * nu;
  if (kStress) {
    const double C = G / (4.0 * kPi * (1.0 - nu));
    const double dx = C * dd[0], dy = C * dd[1], dz = C * dd[2];
    const double zx = z * dx, zy = z * dy, zd = z * dz;
    const double sxx = 2.0 * dx * D.xz + 2.0 * nu * dy * D.yz + dz * (D.zz + k2 * D.yy) -
                       (zx * D.xxx + zy * D.xxy + zd * D.xxz);
    const double syy = 2.0 * nu * dx * D.xz + 2.0 * dy * D.yz + dz * (D.zz + k2 * D.xx) -
                       (zx * D.xyy + zy * D.yyy + zd * D.yyz);
    const double szz = dz * D.zz - (zx * D.xzz + zy * D.yzz + zd * D.zzz);
    const double sxy = (1.0 - nu) * (dx * D.yz + dy * D.xz) - k2 * dz * D.xy -
                       (zx * D.xxy + zy * D.xyy + zd * D.xyz);
    const double sxz = dx * (D.zz + nu * D.yy) - nu * dy * D.xy - (zx * D.xxz + zy * D.xyz + zd * D.xzz);
    const double syz = dy * (D.zz + nu * D.xx) - nu * dx * D.xy - (zx * D.xyz + zy * D.yyz + zd * D.yzz);
    const double S[3][3] = {{sxx, sxy, sxz}, {sxy, syy, syz}, {sxz, syz, szz}};
    double T[3][3];  // S R
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) T[i][j] = S[i][0] * R[j] + S[i][1] * R[3 + j] + S[i][2] * R[6 + j];
    auto g = [&](int i, int j) { return R[i] * T[0][j] + R[3 + i] * T[1][j] + R[6 + i] * T[2][j]; };  // (R^T S R)_ij
    acc[0] += g(0, 0);
    acc[1] += g(1, 1);
    acc[2] += g(2, 2);
    acc[3] += g(0, 1);
    acc[4] += g(0, 2);
    acc[5] += g(1, 2);
  }
  if (kDisp) {
    const double c = 1.0 / (8.0 * kPi * (1.0 - nu)), k1 = 2.0 * (1.0 - nu);
    const double ux = c * dd[0], uy = c * dd[1], uz = c * dd[2];
    const double ul[3] = {
        ux * (k1 * D.z - z * D.xx) - uy * (z * D.xy) - uz * (k2 * D.x + z * D.xz),
        uy * (k1 * D.z - z * D.yy) - ux * (z * D.xy) - uz * (k2 * D.y + z * D.yz),
        ux * (k2 * D.x - z * D.xz) + uy * (k2 * D.y - z * D.yz) + uz * (k1 * D.z - z * D.zz)};
    for (int i = 0; i < 3; i++) acc[6 + i] += R[i] * ul[0] + R[3 + i] * ul[1] + R[6 + i] * ul[2];
  }
}

}  // namespace r0
}  // namespace bw
