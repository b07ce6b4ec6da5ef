// hex8.cuh -- a field on a C3D8 from its trilinear structure,
// x = sum c_ijk xi^i eta^j zeta^k, shared by the recovery and energy kernels.
#pragma once

// The derivatives of one field at the 2 x 2 x 2 Gauss points from its eight
// nodal values v: the seven coefficients by a Hadamard transform (relative to
// node 0, which also keeps the element's distance from the origin out of the
// rounding); along a direction a derivative is the same at both points, so three
// times four values serve the eight points, in D[0..3] d/dxi, D[4..7] d/deta,
// D[8..11] d/dzeta by the signs (-, -) (-, +) (+, -) (+, +) of the other two.
__device__ __forceinline__ void hex8_point_derivatives(const double* v, double* D) {
  const double v0 = v[0];
  const double a1 = v[1] - v0, a2 = v[2] - v0, a3 = v[3] - v0, a4 = v[4] - v0, a5 = v[5] - v0, a6 = v[6] - v0,
               a7 = v[7] - v0;
  // along xi: sums and differences of the edges (eta, zeta) = --, +-, -+, ++
  const double p0 = a1, p1 = a2 + a3, p2 = a5 + a4, p3 = a6 + a7;
  const double d0 = a1, d1 = a2 - a3, d2 = a5 - a4, d3 = a6 - a7;
  const double pe0 = p1 - p0, pe1 = p3 - p2, ps0 = p1 + p0, ps1 = p3 + p2;  // along eta
  const double de0 = d1 - d0, de1 = d3 - d2, ds0 = d1 + d0, ds1 = d3 + d2;
  constexpr double G = 0.57735026918962576451;  // 1 / sqrt(3)
  const double kx = 0.125 * (ds1 + ds0), ky = 0.125 * (pe1 + pe0), kz = 0.125 * (ps1 - ps0);
  // xi eta, xi zeta, eta zeta at |.| = G, xi eta zeta at G^2
  const double kxy = 0.125 * G * (de1 + de0), kxz = 0.125 * G * (ds1 - ds0), kyz = 0.125 * G * (pe1 - pe0),
               kxyz = (1.0 / 24.0) * (de1 - de0);
  // d/dxi = kx + s2 kxy + s3 (kxz + s2 kxyz) and so on
  const double xm = kx - kxy, xp = kx + kxy, xbm = kxz - kxyz, xbp = kxz + kxyz;
  const double ym = ky - kxy, yp = ky + kxy, zm = kz - kxz, zp = kz + kxz, bm = kyz - kxyz, bp = kyz + kxyz;
  D[0] = xm - xbm;
  D[1] = xm + xbm;
  D[2] = xp - xbp;
  D[3] = xp + xbp;
  D[4] = ym - bm;
  D[5] = ym + bm;
  D[6] = yp - bp;
  D[7] = yp + bp;
  D[8] = zm - bm;
  D[9] = zm + bm;
  D[10] = zp - bp;
  D[11] = zp + bp;
}

// point g = 4 [xi > 0] + 2 [eta > 0] + [zeta > 0]: where its derivatives stand in D
__device__ __forceinline__ int hex8_dxi(int g) { return g & 3; }
__device__ __forceinline__ int hex8_deta(int g) { return 4 + (g >> 2) * 2 + (g & 1); }
__device__ __forceinline__ int hex8_dzeta(int g) { return 8 + (g >> 1); }
