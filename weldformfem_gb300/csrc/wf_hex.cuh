// Arithmetic of the hexahedra that the FP64 step and its reverse pass share:
// Walsh sums over the corners and their transposes, the adjugate of 8 J, and
// the hourglass coefficient's power of the volume.
#pragma once

namespace wf {
namespace {

// Walsh sums of the eight nodal values of a hexahedron, weighted by the corner
// signs {-, xi, eta, zeta, eta zeta, xi zeta, xi eta, xi eta zeta} (index 0 is
// not formed): 1..3 are the derivative directions of the trilinear shape
// functions at the centre (8 J for coordinates), 4..7 the hourglass base
// vectors. 23 additions; unused outputs cost nothing.
template <typename T>
__device__ __forceinline__ void walsh8d(const T (&v)[8], T (&o)[8]) {
  const T a0 = v[1] + v[0], b0 = v[1] - v[0];
  const T a1 = v[2] + v[3], b1 = v[2] - v[3];
  const T a2 = v[5] + v[4], b2 = v[5] - v[4];
  const T a3 = v[6] + v[7], b3 = v[6] - v[7];
  const T c0 = a1 + a0, d0 = a1 - a0, e0 = b1 + b0, f0 = b1 - b0;
  const T c1 = a3 + a2, d1 = a3 - a2, e1 = b3 + b2, f1 = b3 - b2;
  o[1] = e1 + e0;
  o[2] = d1 + d0;
  o[3] = c1 - c0;
  o[4] = d1 - d0;
  o[5] = e1 - e0;
  o[6] = f1 + f0;
  o[7] = f1 - f0;
}

// Nodal values of o1 xi + o2 eta + o3 zeta: opposite corners differ in sign,
// so 6 additions give all eight.
template <typename T>
__device__ __forceinline__ void synth_linear(T o1, T o2, T o3, T (&v)[8]) {
  const T p = o3 + o2, m = o3 - o2;
  v[6] = p + o1;
  v[7] = p - o1;
  v[5] = m + o1;
  v[4] = m - o1;
  v[0] = -v[6];
  v[1] = -v[7];
  v[2] = -v[4];
  v[3] = -v[5];
}

// Nodal values of o4 eta zeta + o5 xi zeta + o6 xi eta + o7 xi eta zeta: the
// part even under the inversion of the corner (o4, o5, o6) and the odd one.
template <typename T>
__device__ __forceinline__ void synth_hourglass(T o4, T o5, T o6, T o7, T (&v)[8]) {
  const T s = o4 + o5, d = o4 - o5;
  const T e06 = s + o6, e17 = d - o6;   // corners 0, 6 and 1, 7
  const T e24 = o6 - s, e35 = -d - o6;  // corners 2, 4 and 3, 5
  v[6] = e06 + o7;
  v[0] = e06 - o7;
  v[1] = e17 + o7;
  v[7] = e17 - o7;
  v[4] = e24 + o7;
  v[2] = e24 - o7;
  v[3] = e35 + o7;
  v[5] = e35 - o7;
}

// adj(X) and det(X) of X = 8 J (rows xi, eta, zeta): A[k][m] = cofactor [m][k].
template <typename T>
__device__ __forceinline__ T adjugate8(const T (&X)[3][3], T (&A)[3][3]) {
  A[0][0] = fma(X[1][1], X[2][2], -(X[1][2] * X[2][1]));
  A[1][0] = fma(X[1][2], X[2][0], -(X[1][0] * X[2][2]));
  A[2][0] = fma(X[1][0], X[2][1], -(X[1][1] * X[2][0]));
  A[0][1] = fma(X[0][2], X[2][1], -(X[0][1] * X[2][2]));
  A[1][1] = fma(X[0][0], X[2][2], -(X[0][2] * X[2][0]));
  A[2][1] = fma(X[0][1], X[2][0], -(X[0][0] * X[2][1]));
  A[0][2] = fma(X[0][1], X[1][2], -(X[0][2] * X[1][1]));
  A[1][2] = fma(X[0][2], X[1][0], -(X[0][0] * X[1][2]));
  A[2][2] = fma(X[0][0], X[1][1], -(X[0][1] * X[1][0]));
  return fma(X[0][2], A[2][0], fma(X[0][1], A[1][0], X[0][0] * A[0][0]));
}

// v^0.6666666 (the hourglass coefficient's exponent, test_1el_3D.cpp:185) for
// v > 0, as p (1 + u) with p = v y0 and y0 the FP32 inverse cube root, u of about
// 1e-6 and one rounding at the end: y = y0 (1 + t), t = e / 3 + 2 e^2 / 9 with
// e = 1 - v y0^3 of about 1e-7 (a third-order correction; v y0 in two parts and
// y0^2 exact), v^(2/3) = v y, and v^(0.6666666 - 2/3) = exp(z) with |z| < 5e-6 as
// 1 + z + z^2 / 2. The exponent's difference is its own literal (formed from the
// two doubles it is off by 4e-17), and the logarithm is within 1e-9: of the
// mantissa m = (1 + s) / (1 - s) the series 2 (s + s^3 / 3 + ...) with s in two
// floats, all FP32 (logf alone is 4e-8 off, 4e-15 in the result). At most
// 1.5e-16 relative, as pow's; 17 FP64 instructions; values out of the FP32 range
// take pow.
__device__ __forceinline__ double pow_two_thirds(double v) {
  if (!(v > 1e-30 && v < 1e30)) return pow(v, 0.6666666);
  const double y0 = (double)rcbrtf((float)v);
  const double p = v * y0, pe = fma(v, y0, -p), y2 = y0 * y0;
  const double e = fma(-pe, y2, fma(-p, y2, 1.0));
  const double t = e * fma(e, 2.0 / 9.0, 1.0 / 3.0);
  // v = m 2^q with m in [0.7, 1.42)
  const int hi = __double2hiint(v);
  const double md = __hiloint2double(0x3ff00000 | (hi & 0xfffff), __double2loint(v));
  int q = (hi >> 20) - 1023;
  float m = (float)md, ml = (float)(md - (double)m);
  if (m > 1.4142f) {
    m *= 0.5f;
    ml *= 0.5f;
    q += 1;
  }
  // s = (m + ml - 1) / (m + ml + 1) = a + al; the differences are exact
  const float n = m - 1.0f, d = m + 1.0f, dl = (m - (d - 1.0f)) + ml;
  const float a = n / d, al = (fmaf(-a, d, n) + fmaf(-a, dl, ml)) / d;
  const float w = a * a;
  const float c = fmaf(w, fmaf(w, fmaf(w, fmaf(w, 1.f / 11, 1.f / 9), 1.f / 7), 0.2f), 1.f / 3);
  const float rest = 2.0f * fmaf(a * w, c, fmaf(w, al, al));
  const double ln = fma((double)q, 0.693147180559945309, (double)(2.0f * a) + (double)rest);
  const double z = -6.666666666858372e-08 * ln, x = fma(0.5 * z, z, z);
  return p + fma(p, fma(t, x, t) + x, pe);
}

// X[m][k] = sum of the corners' coordinates k weighted by the sign of
// direction m (8 J), from differences along the edges (21 additions a
// component; the velocity sums take 17). The pressure is the bulk modulus
// times a change of volume of 1e-3 and less, so the rounding of these sums shows
// in the state. Which form is closer depends on what it is held against: 1.05 M
// hexahedra, 20 steps, displacement 2e-13 from edge differences and 8e-13 from the
// reference's alternating sums against 64-bit sums of coordinates relative to a
// corner, 2e-12 and 6e-13 against 64-bit alternating sums, which share the latter's
// rounding. Against 80-bit arithmetic (8^3 and 16^3 cubes, 64 steps) the two are
// alike, 7.3e-13 and 7.4e-13, 8.2e-13 and 8.9e-13.
template <typename T>
__device__ __forceinline__ void corner_sums(const T (&x2)[8][3], T (&X)[3][3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    T v[8];
#pragma unroll
    for (int a = 0; a < 8; a++) v[a] = x2[a][k];
    X[0][k] = ((v[1] - v[0]) + (v[2] - v[3])) + ((v[5] - v[4]) + (v[6] - v[7]));
    X[1][k] = ((v[2] - v[1]) + (v[3] - v[0])) + ((v[6] - v[5]) + (v[7] - v[4]));
    X[2][k] = ((v[4] - v[0]) + (v[6] - v[2])) + ((v[5] - v[1]) + (v[7] - v[3]));
  }
}

}  // namespace
}  // namespace wf
