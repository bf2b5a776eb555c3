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
// v > 0: the inverse cube root from its FP32 value by one third-order
// correction, y (1 + e / 3 + 2 e^2 / 9) with e = 1 - v y^3 of about 1e-7, then
// v^(2/3) = v y, and v^(0.6666666 - 2/3) = exp(z) with |z| < 5e-6 as
// 1 + z + z^2 / 2; in z the logarithm of the mantissa is FP32 (3e-8 absolute,
// 2e-15 in the result). About 15 FP64 instructions; values out of the FP32
// range take pow.
__device__ __forceinline__ double pow_two_thirds(double v) {
  if (!(v > 1e-30 && v < 1e30)) return pow(v, 0.6666666);
  const double y0 = (double)rcbrtf((float)v);
  const double e = fma(-(v * y0), y0 * y0, 1.0);
  const double y = fma(y0 * e, fma(e, 2.0 / 9.0, 1.0 / 3.0), y0);
  // v = m 2^q with m in [1, 2): ln m from its FP32 rounding and the rest
  const int hi = __double2hiint(v);
  const double md = __hiloint2double(0x3ff00000 | (hi & 0xfffff), __double2loint(v));
  const float m = (float)md;
  const double ln = fma((double)((hi >> 20) - 1023), 0.693147180559945309,
                        (double)logf(m) + (double)((float)(md - (double)m) / m));
  const double z = (0.6666666 - 2.0 / 3.0) * ln;
  return (v * y) * fma(z, fma(z, 0.5, 1.0), 1.0);
}

// X[m][k] = sum of the corners' coordinates k weighted by the sign of
// direction m (8 J), from differences along the edges (21 additions a
// component; the velocity sums take 17). The pressure is the bulk modulus
// times a change of volume of 1e-3 and less, and differences of sums of
// absolute coordinates left the step's largest rounding error (against 64-bit
// sums of coordinates relative to a corner, 1.05 M hexahedra, 20 steps:
// displacement 2e-13 from edge differences, 8e-13 without, as the reference's
// alternating sums).
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
