// FP64 step kernels.
//
// This translation unit is compiled with --fmad=false: tetrahedra run the
// reference's arithmetic operation for operation and round exactly as the
// reference CPU code does with FMA contraction off (the reference build passes
// --fmad=false to nvcc, src/common/CMakeLists.txt:16). Hexahedra compute the
// same quantities in fewer operations (k_fp64_hexes), with explicit FMA, and
// stay within 1e-9 of the reference. One step is four launches:
//   geometry  (element): J, detJ, volume             -> vol
//   nodal     (node)   : volume sums, lumped mass, J ratio
//   elements  (element): dN, D/W, pressure, Jaumann + radial return,
//                        B^T sigma, hourglass        -> element forces
//   nodes     (node)   : deterministic gather of element forces over the
//                        node->element lists, contact, acceleration, BCs,
//                        Chung-Hulbert corrector, position update and the
//                        next step's predictor; reaction sum (last block).
#include "wf_hex.cuh"
#include "wf_internal.cuh"
#include "wf_trimesh.cuh"

namespace wf {
namespace {

constexpr int kElemThreads = 128;
constexpr int kNodeThreads = 256;

__device__ __forceinline__ double det3(const double J[3][3]) {
  // Matrix::calcDet (include/common/Matrix.h:593-620)
  return J[0][0] * J[1][1] * J[2][2] - J[0][0] * J[1][2] * J[2][1] -
         J[0][1] * J[1][0] * J[2][2] + J[0][1] * J[1][2] * J[2][0] +
         J[0][2] * J[1][0] * J[2][1] - J[0][2] * J[1][1] * J[2][0];
}

// Jacobian of a tetrahedron from its node coordinates (Domain_d.C:1866-1870).
__device__ __forceinline__ void jacobian(const double (&x2)[4][3], double J[3][3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    J[0][k] = x2[1][k] - x2[0][k];
    J[1][k] = x2[2][k] - x2[0][k];
    J[2][k] = x2[3][k] - x2[0][k];
  }
}

// Adjugate of J (AdjMat, Matrix.h:694-727), inv[k][m].
__device__ __forceinline__ void adjugate(const double J[3][3], double inv[3][3]) {
  inv[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]);
  inv[1][0] = -(J[1][0] * J[2][2] - J[1][2] * J[2][0]);
  inv[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
  inv[0][1] = -(J[0][1] * J[2][2] - J[0][2] * J[2][1]);
  inv[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]);
  inv[2][1] = -(J[0][0] * J[2][1] - J[0][1] * J[2][0]);
  inv[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]);
  inv[1][2] = -(J[0][0] * J[1][2] - J[0][2] * J[1][0]);
  inv[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]);
}

template <int NPE>
__device__ __forceinline__ double weight() {
  return NPE == 8 ? 8.0 : 1.0 / 6.0;
}

template <int NPE>
__device__ __forceinline__ void gather_x(const StepParams &P, const double *x, int64_t e,
                                         double (&x2)[NPE][3], int32_t (&nid)[NPE]) {
#pragma unroll
  for (int a = 0; a < NPE; a++) nid[a] = __ldg(&P.elnod[a * P.ne + e]);
#pragma unroll
  for (int a = 0; a < NPE; a++) {
    x2[a][0] = __ldg(&x[nid[a]]);
    x2[a][1] = __ldg(&x[P.np + nid[a]]);
    x2[a][2] = __ldg(&x[2 * P.np + nid[a]]);
  }
}

// ---------------------------------------------------------------------------
// geometry: vol = 0.0 + detJ * w * 1.0 (Mechanical.C:264-293), and the adjugate
// of the Jacobian (of 8 J for hexahedra) for the element kernel of the step:
// 72 bytes written and read once cost less than the 70 FP64 instructions that
// form it again (1.05 M hexahedra: element kernel 805 -> 662 us, this one
// 150 -> 152 us).
template <int NPE>
__global__ void __launch_bounds__(kElemThreads) k_fp64_geometry(StepParams P, Fp64State S,
                                                           int store_detj) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P.ne) return;
  double x2[NPE][3];
  int32_t nid[NPE];
  gather_x<NPE>(P, S.x, e, x2, nid);
  double J[3][3], A[3][3], detJ, v;
  if constexpr (NPE == 8) {
    corner_sums(x2, J);
    detJ = adjugate8(J, A) * (1.0 / 512.0);
    v = detJ * 8.0;
  } else {
    jacobian(x2, J);
    detJ = det3(J);
    v = 0.0;
    v += detJ * weight<NPE>() * 1.0;
  }
  S.vol[e] = v;
  if (store_detj) S.detJ[e] = detJ;
  if (!S.adj) return;   // the preamble, or a detJ readback
  if constexpr (NPE == 4) adjugate(J, A);
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int m = 0; m < 3; m++) S.adj[(3 * k + m) * P.ne + e] = A[k][m];
  if constexpr (NPE == 4) S.adj[9 * P.ne + e] = detJ;
}

// ---------------------------------------------------------------------------
// nodal: CalcNodalVol (Mechanical.C:1555-1572), CalcNodalMassFromVol
// (:1576-1601) and the nodal volume ratio of calcElemPressure (:694-705).
// init_mode 1 also forms the constant sum of initial volumes.
template <int NPE>
__global__ void __launch_bounds__(kNodeThreads) k_fp64_nodal(StepParams P, Fp64State S,
                                                        int init_mode) {
  int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.nn) return;
  const int32_t b = __ldg(&P.off[n]), c = __ldg(&P.off[n + 1]) - b;
  auto elem = [&](int32_t k) -> int32_t { return __ldg(&P.slot[b + k]) / NPE; };
  // sums in list order, eight entries at a time: a chunk's loads are in
  // flight together
  double s = 0.0, s0 = 0.0;
  for (int32_t k0 = 0; k0 < c; k0 += 8) {
    double g[8], g0[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int32_t e = (k0 + j < c) ? elem(k0 + j) : -1;
      g[j] = (e >= 0) ? __ldg(&S.vol[e]) : 0.0;
      g0[j] = (init_mode && e >= 0) ? __ldg(&S.vol0[e]) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) s += g[j];
    if (init_mode) {
#pragma unroll
      for (int j = 0; j < 8; j++) s0 += g0[j];
    }
  }
  if (init_mode) S.s0[n] = s0;
  else s0 = S.s0[n];
  double voln = s;
  voln /= NPE;
  S.voln[n] = voln;
  if (P.mass_mode == 0 || init_mode) {
    // sum of rho_e voln / c over the node's elements. The densities of a mesh
    // of one material differ in their last bits (rho_0 vol_0 / vol_0), so
    // every entry needs its own quotient: FP64 divisions at about ten FP64
    // instructions each.
    double mass = 0.0, rs = 0.0;
    const double dc = c, rc = 1.0 / dc;
    for (int32_t k0 = 0; k0 < c; k0 += 8) {
      double g[8];
#pragma unroll
      for (int j = 0; j < 8; j++) g[j] = (k0 + j < c) ? __ldg(&S.rho[elem(k0 + j)]) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if constexpr (NPE == 8) {
          rs += g[j];
        } else {
          // the reference's sum in list order, bit for bit: x / c as q = x (1 / c)
          // corrected by its remainder, correctly rounded when 1 / c is
          // (Markstein's theorem; x / c for c up to 4096 checked on random x)
          const double x = g[j] * voln;
          const double q = x * rc;
          mass += fma(fma(-q, dc, x), rc, q);
        }
      }
    }
    // hexahedra: the densities' sum times voln / c, an exact division for the
    // 1, 2, 4 or 8 elements of a box mesh's nodes
    if constexpr (NPE == 8) mass = c > 0 ? rs * voln * rc : 0.0;
    // tetrahedra: an infinity has no remainder, and zero times it is not zero
    if (NPE == 4 && !(fabs(voln) < 1e290)) {
      mass = 0.0;
      for (int32_t k = 0; k < c; k++) mass += __ldg(&S.rho[elem(k)]) * voln / c;
    }
    S.mass[n] = mass;
  }
  S.jr[n] = s / s0;
}

// GMT law (CalcGMTYieldStress and CalcGMTTangentModulus, Material.cuh:417-478)
// in FP64: strain e, strain rate r and temperature T clamped to the
// material's ranges, then the reference's products in its order; mp points to
// the material in global memory. Not inlined: the law's temporaries stay out
// of the element kernel's register budget.
static __device__ __noinline__ double gmt_sy(double e, double r, double T, const MatDev *mp) {
  const MatDev &m = *mp;
  e = clamp_range(e, m.g_emin, m.g_emax);
  r = clamp_range(r, m.g_rmin, m.g_rmax);
  T = clamp_range(T, m.g_Tmin, m.g_Tmax);
  return m.g_C1 * exp(m.g_C2 * T) * pow(e, m.g_n1 * T + m.g_n2) * exp((m.g_I1 * T + m.g_I2) / e) *
         pow(r, m.g_m1 * T + m.g_m2);
}
static __device__ __noinline__ double gmt_et(double e, double r, double T, const MatDev *mp) {
  const MatDev &m = *mp;
  e = clamp_range(e, m.g_emin, m.g_emax);
  r = clamp_range(r, m.g_rmin, m.g_rmax);
  T = clamp_range(T, m.g_Tmin, m.g_Tmax);
  return m.g_C1 * exp(m.g_C2 * T) * pow(r, m.g_m1 * T + m.g_m2) * pow(e, T * m.g_n1 + m.g_n2 - 2.0) *
         (-m.g_I1 * T - m.g_I2 + e * (m.g_n1 * T + m.g_n2)) * exp((m.g_I1 * T + m.g_I2) / e);
}

__device__ __forceinline__ double hollomon_sy(double strain, const MatDev &m) {
  if (strain + m.eps0 > m.eps1) return m.hol_K * pow(strain + m.eps0, m.hol_m);
  return m.sy0;
}
__device__ __forceinline__ double hollomon_et(double strain, const MatDev &m) {
  if (strain + m.eps0 > m.eps1) return m.hol_K * m.hol_m * pow(strain + m.eps0, (m.hol_m - 1.0));
  return 0.;
}

// Element pressure: calcElemPressure (Mechanical.C:691-819) from the mean of
// the nodes' J ratios, or calcElemPressureANP (:1220-1250). div_v is the
// divergence of the predicted velocity times detJ (stabilisation only).
template <int NPE>
__device__ __forceinline__ double element_pressure(const StepParams &P, const Fp64State &S,
                                                   const MatDev &m, int64_t e,
                                                   const int32_t (&nid)[NPE], double vol,
                                                   double div_v) {
  double p;
  if (P.press_alg == 1) {
    p = S.p[e];
    for (int a = 0; a < NPE; a++) p += P.k0 * (1.0 - __ldg(&S.jr[nid[a]]));
    p *= 0.25 * NPE;
    return p;
  }
  const double K = m.K;
  double J_avg = 0.0;
#pragma unroll
  for (int a = 0; a < NPE; a++) J_avg += __ldg(&S.jr[nid[a]]);
  J_avg /= NPE;
  if (!P.stab_on) {
    // All stabilisation parameters zero: J_bar = 0 * J_local + 1 * J_avg
    // = J_avg and the 0 * log(J_bar) term adds only a signed zero.
    double J_bar = J_avg;
    if (J_bar < 0.0) J_bar = 0.2;
    return -K * (J_bar - 1.0);
  }
  const double J_local = vol / __ldg(&S.vol0[e]);
  const double *st = P.stab;
  const double rho_e = S.rho[e];
  const double h = pow(vol, 1.0 / 3.0);
  bool is_contact = false;
  if (P.contact) {
    for (int a = 0; a < NPE; a++) {
      double c0 = S.cf[nid[a]], c1 = S.cf[P.np + nid[a]], c2 = S.cf[2 * P.np + nid[a]];
      if (c0 * c0 + c1 * c1 + c2 * c2 > 0) { is_contact = true; break; }
    }
  }
  double alpha = is_contact ? st[1] : st[0];
  double J_bar = alpha * J_local + (1 - alpha) * J_avg;
  if (J_bar < st[9]) J_bar = 0.2;
  double p_physical = -K * (st[6] * log(J_bar) + (1.0 - st[6]) * (J_bar - 1.0));
  double c = sqrt(K / rho_e);
  double tau = h / (2.0 * c);
  double p_pspg = 0.0;
  double p_hg = (is_contact ? st[3] : st[2]) * K * fabs(J_local - J_avg);
  double p_q = 0.0;
  if (div_v < 0.0) {
    double t1 = st[7] * tau * div_v * K, t2 = st[8] * K;
    p_pspg = (t2 < t1) ? t2 : t1;
    double q1 = st[4] * rho_e * h * c * (-div_v);
    double delta_J = 1.0 - J_local;
    double q2 = st[5] * K * delta_J;
    p_q = is_contact ? 0.5 * (q1 + q2) : ((q1 < q2) ? q2 : q1);
  }
  p = p_physical + p_pspg + p_hg + p_q;
  return p;
}

// Yield stress and tangent modulus of the element's law. eff, jTh and temp
// carry what the rate-dependent laws share between the two.
struct LawState {
  double eff, jTh, temp;
};
template <int NPE, bool TH>
__device__ __forceinline__ double yield_stress(const StepParams &P, const Fp64State &S,
                                               const MatDev &m, int32_t mat_id,
                                               const int32_t (&nid)[NPE], double pls, double s00,
                                               double s11, double s22, double s01, double s12,
                                               double s02, LawState &w) {
  w.eff = 0.0;
  w.jTh = m.jc_Th;
  w.temp = m.g_T;  // GMT element temperature
  if (m.model == WF_MAT_JOHNSON_COOK || m.model == WF_MAT_GMT) {
    // effective strain rate (Mechanical.C:1701-1705)
    w.eff = sqrt(0.5 * ((s00 - s11) * (s00 - s11) + (s11 - s22) * (s11 - s22) +
                        (s22 - s00) * (s22 - s00)) +
                 3.0 * (s01 * s01 + s12 * s12 + s02 * s02));
    if constexpr (TH) {
      // element temperature: mean of its node temperatures (the reference
      // reads T[e], a node array indexed by element)
      double ts = 0.0;
#pragma unroll
      for (int a = 0; a < NPE; a++) ts += S.T[nid[a]];
      w.temp = ts / NPE;
      if (m.model == WF_MAT_JOHNSON_COOK)
        w.jTh = 1.0 - pow((w.temp - m.jc_Tt) / (m.jc_Tm - m.jc_Tt), m.jc_m);
    }
    if (m.model == WF_MAT_JOHNSON_COOK) {
      // CalcJohnsonCookYieldStress (Material.cuh:377-392)
      const double sr = (w.eff == 0.0) ? 1.e-5 : w.eff;
      return (m.sy0 + m.jc_B * pow(pls, m.jc_n)) * (1.0 + m.jc_C * log(sr / m.jc_eps0)) * w.jTh;
    }
    return gmt_sy(pls, w.eff, w.temp, P.mats + mat_id);
  }
  if (m.model == WF_MAT_HOLLOMON) return hollomon_sy(pls, m);
  return m.sy0 + m.H * pls;
}
__device__ __forceinline__ double tangent_modulus(const StepParams &P, const MatDev &m,
                                                  int32_t mat_id, double pls,
                                                  const LawState &w) {
  if (m.model == WF_MAT_JOHNSON_COOK) {
    // CalcJohnsonCookTangentModulus (Material.cuh:397-410) at min(edot, m_max_edot)
    const double er = (P.max_edot < w.eff) ? P.max_edot : w.eff;
    return (pls > 0.) ? m.jc_n * m.jc_B * pow(pls, m.jc_n - 1.) *
                            (1.0 + m.jc_C * log(er / m.jc_eps0)) * w.jTh
                      : m.E * 0.1;
  }
  if (m.model == WF_MAT_GMT)
    return gmt_et(pls, (P.max_edot < w.eff) ? P.max_edot : w.eff, w.temp, P.mats + mat_id);
  return (m.model == WF_MAT_HOLLOMON) ? hollomon_et(pls, m) : m.H;
}

// Plastic heat (Mechanical.C:1783-1810): m_plheatfraction sigma : (d eps_p / dt),
// the plastic strain increment along the returned stress, shear terms doubled.
__device__ __forceinline__ double plastic_heat(const StepParams &P, const double (&SG)[6],
                                               double dep, double sy, double dt) {
  // sigma : increment with the increment (3/2) dep / sy dev(sigma) written out
  const double a = SG[0] - SG[1], b = SG[1] - SG[2], c = SG[2] - SG[0];
  const double nn = 0.5 * fma(a, a, fma(b, b, c * c));
  const double ss = fma(SG[3], SG[3], fma(SG[4], SG[4], SG[5] * SG[5]));
  return P.plheat_frac * (nn + 3.0 * ss) * dep / (sy * dt);
}

// Artificial viscosity (calcArtificialViscosity, Mechanical.C:1948-1977; serial
// in the reference, per element here).
__device__ __forceinline__ void add_viscosity(const StepParams &P, const Fp64State &S,
                                              const MatDev &m, int64_t e, double eps_v, double vol,
                                              double (&SG)[6]) {
  const double c = sqrt(m.K / S.rho[e]);
  if (fabs(eps_v) > 1e-12) {
    const double l = pow(vol, 1.0 / 3.0);
    double q = P.av[0] * c * fabs(eps_v) * l + P.av[1] * pow(eps_v * l, 2);
    q = (1e9 < q) ? 1e9 : q;
    const double qs = (eps_v > 0) ? -q : q;
    SG[0] += qs;
    SG[1] += qs;
    SG[2] += qs;
  }
}

// calcThermalExpansion (Thermal.C:163-178): exp_T times the mean of the
// previous step's element-node temperature rates, read at the element's node
// ids as the reference indexes them.
template <int NPE>
__device__ __forceinline__ double thermal_strain_rate(const StepParams &P, const Fp64State &S,
                                                      const MatDev &m, const int32_t (&nid)[NPE],
                                                      long long step) {
  const double *prev = S.dte + ((step + 1) & 1) * P.ne * NPE;
  double g = 0.0;
#pragma unroll
  for (int a = 0; a < NPE; a++) g += 1.0 / NPE * prev[nid[a]];
  return m.exp_T * g;
}

// Element-node temperature rates (Domain_d::ThermalCalcs, Thermal.C:27-106):
// -(K T)_a / m_a plus the plastic heat 0.9 q vol split evenly over the nodes
// over m_a cp; KT = (K T)_a. One division per node.
template <int NPE>
__device__ __forceinline__ void store_temperature_rates(const StepParams &P, const Fp64State &S,
                                                        const MatDev &m, int64_t e,
                                                        const int32_t (&nid)[NPE], long long step,
                                                        const double (&KT)[NPE], double q_pl,
                                                        double vol) {
  double *cur = S.dte + (step & 1) * P.ne * NPE + e * NPE;
  const double heat = 0.9 * q_pl * vol / NPE / m.cp_T;
#pragma unroll
  for (int a = 0; a < NPE; a++) cur[a] = (heat - KT[a]) / S.mass[nid[a]];
}

// The stress part of an element in FMA form (hexahedra, and tetrahedra with
// thermal coupling): Jaumann rate, radial return, artificial viscosity; writes
// the element's fields and returns sigma in SG and the plastic heat. In: the
// strain rate, the spin and the pressure. The reference's yy and zz Jaumann
// terms are (a - b) + (b - a), exactly zero.
template <int NPE, bool TH>
__device__ __forceinline__ void stress_step(const StepParams &P, const Fp64State &S,
                                            const MatDev &m, int32_t mat_id, int64_t e,
                                            const int32_t (&nid)[NPE], double s00, double s11,
                                            double s22, double s01, double s12, double s02,
                                            double w01, double w12, double w02, double p,
                                            double vol, double (&SG)[6], double &q_pl) {
  const int64_t ne = P.ne;
  // Jaumann rate with the reference's product, then the radial return; the
  // pressure drops out of the trial stress's deviator
  const double dt = P.espec ? P.spec_dt[P.espec[e]] : P.dt;
  double t0 = S.tau[e], t1 = S.tau[ne + e], t2 = S.tau[2 * ne + e];
  double t3 = S.tau[3 * ne + e], t4 = S.tau[4 * ne + e], t5 = S.tau[5 * ne + e];
  {
    const double g2 = 2.0 * m.G * dt;
    const double c = (1.0 / 3.0) * (s00 + s11 + s22);
    const double q0 = 2.0 * fma(t3, w01, t5 * w02);
    const double q3 = fma(w01, t0 + t1, fma(w02, t4, -(t5 * w12)));
    const double q4 = fma(w12, t1 + t2, fma(w02, t3, -(t5 * w01)));
    const double q5 = fma(w02, t0 + t2, fma(w12, t3, w01 * t4));
    t0 = fma(q0, dt, fma(s00 - c, g2, t0));
    t1 = fma(s11 - c, g2, t1);
    t2 = fma(s22 - c, g2, t2);
    t3 = fma(q3, dt, fma(s01, g2, t3));
    t4 = fma(q4, dt, fma(s12, g2, t4));
    t5 = fma(q5, dt, fma(s02, g2, t5));
  }
  const double tm = (1.0 / 3.0) * (t0 + t1 + t2);
  const double d0s = t0 - tm, d1s = t1 - tm, d2s = t2 - tm;
  // sig_trial^2 = 3 J2
  const double q2 = 1.5 * fma(d0s, d0s, fma(d1s, d1s, fma(d2s, d2s,
                          2.0 * fma(t3, t3, fma(t4, t4, t5 * t5)))));
  double pls = S.pls[e];
  LawState law;
  const double sy = yield_stress<NPE, TH>(P, S, m, mat_id, nid, pls, s00, s11, s22, s01, s12, s02,
                                          law);
  double dep = 0.0;
  // sy < sig_trial, without the square root for elements well inside the
  // yield surface (a NaN enters and fails the exact test, as sy < NaN does)
  if (sy < 0.0 || !(q2 < sy * sy)) {
    // (0 and infinity keep the square root's value)
    const double rs = rsqrt(q2), sig_trial = (q2 > 0.0 && !isinf(q2)) ? q2 * rs : q2;
    if (sy < sig_trial) {
      const double G3 = 3.0 * m.G;
      const double dgamma = (m.model == WF_MAT_BILINEAR)
                                ? (sig_trial - sy) * m.i3GH
                                : (sig_trial - sy) / (G3 + tangent_modulus(P, m, mat_id, pls, law));
      const double factor = 1.0 - (G3 * dgamma) * rs;
      t0 = d0s * factor; t1 = d1s * factor; t2 = d2s * factor;
      t3 = t3 * factor; t4 = t4 * factor; t5 = t5 * factor;
      pls += dgamma;
      dep = dgamma;
    }
  }
  SG[0] = t0 - p; SG[1] = t1 - p; SG[2] = t2 - p;
  SG[3] = t3; SG[4] = t4; SG[5] = t5;
  q_pl = 0.0;
  if (TH && dep > 0.0) q_pl = plastic_heat(P, SG, dep, sy, dt);
  S.eps[e] = fma(s00, dt, S.eps[e]);
  S.eps[ne + e] = fma(s11, dt, S.eps[ne + e]);
  S.eps[2 * ne + e] = fma(s22, dt, S.eps[2 * ne + e]);
  S.eps[3 * ne + e] = fma(s01, dt, S.eps[3 * ne + e]);
  S.eps[4 * ne + e] = fma(s12, dt, S.eps[4 * ne + e]);
  S.eps[5 * ne + e] = fma(s02, dt, S.eps[5 * ne + e]);
  if (P.av_on) add_viscosity(P, S, m, e, s00 + s11 + s22, vol, SG);
  S.p[e] = p;
  S.pls[e] = pls;
  S.sy[e] = sy;
#pragma unroll
  for (int c = 0; c < 6; c++) S.sig[c * ne + e] = SG[c];
  S.tau[e] = t0; S.tau[ne + e] = t1; S.tau[2 * ne + e] = t2;
  S.tau[3 * ne + e] = t3; S.tau[4 * ne + e] = t4; S.tau[5 * ne + e] = t5;
  S.sr[e] = s00; S.sr[ne + e] = s11; S.sr[2 * ne + e] = s22;
  S.sr[3 * ne + e] = s01; S.sr[4 * ne + e] = s12; S.sr[5 * ne + e] = s02;
  // the spin's diagonal stays zero (rows 0..2 are never written)
  S.rr[3 * ne + e] = w01; S.rr[4 * ne + e] = w12; S.rr[5 * ne + e] = w02;
}

// ---------------------------------------------------------------------------
// elements: calcElemJAndDerivatives, calcElemStrainRates (Mechanical.C:41-126),
// calcElemPressure (:691-819) or calcElemPressureANP (:1220-1250),
// CalcStressStrain (:1664-1839), calcArtificialViscosity (:1948-1977),
// calcElemForces (:375-481) and the 3-D viscous hourglass forces.
// TH: thermal coupling (a separate instantiation keeps the common case's
// register allocation). Element forces go to fe[(a * 3 + k) * ne + e] (and the
// hourglass forces to fhg likewise): neighbouring threads store neighbouring
// values, and the node gather reads them so.
//
// Tetrahedra: the reference's operations in its order (FMA contraction off),
// bit for bit the reference's forces.
__global__ void __launch_bounds__(kElemThreads) k_fp64_tets(StepParams P, Fp64State S) {
  constexpr int NPE = 4;
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P.ne) return;
  const int64_t ne = P.ne;
  int32_t nid[NPE];
#pragma unroll
  for (int a = 0; a < NPE; a++) nid[a] = __ldg(&P.elnod[a * ne + e]);
  // dN/dx detJ (Domain_d.C:1881-1887) from the step's adjugate
  double dH[3][NPE];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double a0 = S.adj[(3 * k) * ne + e], a1 = S.adj[(3 * k + 1) * ne + e],
                 a2 = S.adj[(3 * k + 2) * ne + e];
    dH[k][0] = -a0 - a1 - a2;
    dH[k][1] = a0;
    dH[k][2] = a1;
    dH[k][3] = a2;
  }
  const double detJ = S.adj[9 * ne + e];
  const double vol = __ldg(&S.vol[e]);
  const int32_t mat_id = P.emat ? __ldg(&P.emat[e]) : 0;
  const MatDev m = P.mats[mat_id];

  // strain rate and spin (str_rate / rot_rate, upper triangle)
  double s00 = 0.0, s11 = 0.0, s22 = 0.0, s01 = 0.0, s12 = 0.0, s02 = 0.0;
  double w01 = 0.0, w12 = 0.0, w02 = 0.0;
  double div_v = 0.0;
  const double f = 1.0 / detJ;
#pragma unroll
  for (int a = 0; a < NPE; a++) {
    const double v0 = __ldg(&S.vp[nid[a]]);
    const double v1 = __ldg(&S.vp[P.np + nid[a]]);
    const double v2 = __ldg(&S.vp[2 * P.np + nid[a]]);
    const double d0 = dH[0][a], d1 = dH[1][a], d2 = dH[2][a];
    s00 = s00 + d0 * f * v0;
    s11 = s11 + d1 * f * v1;
    s22 = s22 + d2 * f * v2;
    s01 = s01 + f * (d1 * v0 + d0 * v1);
    w01 = w01 + f * (d1 * v0 - d0 * v1);
    s12 = s12 + f * (d2 * v1 + d1 * v2);
    s02 = s02 + f * (d2 * v0 + d0 * v2);
    w12 = w12 + f * (d2 * v1 - d1 * v2);
    w02 = w02 + f * (d2 * v0 - d0 * v2);
    if (P.stab_on) div_v += d0 * v0 + d1 * v1 + d2 * v2;
  }
  s01 = s01 * 0.5; s02 = s02 * 0.5; s12 = s12 * 0.5;
  w01 = w01 * 0.5; w02 = w02 * 0.5; w12 = w12 * 0.5;
  const double p = element_pressure(P, S, m, e, nid, vol, div_v);

  // Jaumann rate + radial return (CalcStressStrain). The tensor3 algebra of
  // the reference (Tensor3.C) written out on the six stored components: the
  // addends that multiply an exact zero of the spin or of the identity's
  // off-diagonal are dropped, which leaves every value unchanged (only the
  // sign of an exact zero could differ) and saves FP64 instructions.
  const double dt = P.espec ? P.spec_dt[P.espec[e]] : P.dt;
  double t0 = S.tau[e], t1 = S.tau[ne + e], t2 = S.tau[2 * ne + e];
  double t3 = S.tau[3 * ne + e], t4 = S.tau[4 * ne + e], t5 = S.tau[5 * ne + e];
  {
    // SRT = tau * Trans(W), RS = W * tau with the product of Tensor3.C:290-303
    const double srt0 = t3 * w01 + t5 * w02;    // xx
    const double srt1 = t3 * w01 - t4 * w12;    // yy
    const double srt2 = t5 * w02 + t4 * w12;    // zz
    const double srt3 = t0 * w01 - t5 * w12;    // xy
    const double srt4 = t3 * w02 + t1 * w12;    // yz
    const double srt5 = t0 * w02 + t3 * w12;    // xz
    const double rs0 = w01 * t3 + w02 * t5;
    const double rs1 = w12 * t4 - w01 * t3;
    const double rs2 = -(w02 * t5 + w12 * t4);
    const double rs3 = w01 * t1 + w02 * t4;
    const double rs4 = w12 * t2 - w01 * t5;
    const double rs5 = w01 * t4 + w02 * t2;
    const double c = 1.0 / 3.0 * (s00 + s11 + s22);
    const double g2 = 2.0 * m.G;
    t0 = t0 + (((s00 - c) * g2 + srt0) + rs0) * dt;
    t1 = t1 + (((s11 - c) * g2 + srt1) + rs1) * dt;
    t2 = t2 + (((s22 - c) * g2 + srt2) + rs2) * dt;
    t3 = t3 + ((s01 * g2 + srt3) + rs3) * dt;
    t4 = t4 + ((s12 * g2 + srt4) + rs4) * dt;
    t5 = t5 + ((s02 * g2 + srt5) + rs5) * dt;
  }
  // sigma_trial = -p I + tau; s_trial = sigma_trial - tr/3 I
  const double st0 = t0 - p, st1 = t1 - p, st2 = t2 - p;
  const double c2 = (1.0 / 3.0) * (st0 + st1 + st2);
  const double d0s = st0 - c2, d1s = st1 - c2, d2s = st2 - c2;
  const double J2 = 0.5 * (d0s * d0s + 2.0 * t3 * t3 + 2.0 * t5 * t5 + d1s * d1s +
                           2.0 * t4 * t4 + d2s * d2s);
  const double sig_trial = sqrt(3.0 * J2);
  double pls = S.pls[e];
  LawState law;
  const double sy = yield_stress<NPE, false>(P, S, m, mat_id, nid, pls, s00, s11, s22, s01, s12, s02,
                                          law);
  if (sy < sig_trial) {
    const double H = tangent_modulus(P, m, mat_id, pls, law);
    const double G = m.G;
    const double dgamma = (sig_trial - sy) / (3.0 * G + H);
    const double factor = 1.0 - (3.0 * G * dgamma) / sig_trial;
    t0 = d0s * factor; t1 = d1s * factor; t2 = d2s * factor;
    t3 = t3 * factor; t4 = t4 * factor; t5 = t5 * factor;
    pls += dgamma;
  }
  double SG[6] = {t0 - p, t1 - p, t2 - p, t3, t4, t5};
  // total strain: eps = eps + dt * D
  {
    double e0 = S.eps[e], e1 = S.eps[ne + e], e2 = S.eps[2 * ne + e];
    double e3 = S.eps[3 * ne + e], e4 = S.eps[4 * ne + e], e5 = S.eps[5 * ne + e];
    S.eps[e] = e0 + s00 * dt;
    S.eps[ne + e] = e1 + s11 * dt;
    S.eps[2 * ne + e] = e2 + s22 * dt;
    S.eps[3 * ne + e] = e3 + s01 * dt;
    S.eps[4 * ne + e] = e4 + s12 * dt;
    S.eps[5 * ne + e] = e5 + s02 * dt;
  }
  if (P.av_on) add_viscosity(P, S, m, e, s00 + s11 + s22, vol, SG);
  S.p[e] = p;
  S.pls[e] = pls;
  S.sy[e] = sy;
  const double sg0 = SG[0], sg1 = SG[1], sg2 = SG[2], sg3 = SG[3], sg4 = SG[4], sg5 = SG[5];
  S.sig[e] = sg0; S.sig[ne + e] = sg1; S.sig[2 * ne + e] = sg2;
  S.sig[3 * ne + e] = sg3; S.sig[4 * ne + e] = sg4; S.sig[5 * ne + e] = sg5;
  S.tau[e] = t0; S.tau[ne + e] = t1; S.tau[2 * ne + e] = t2;
  S.tau[3 * ne + e] = t3; S.tau[4 * ne + e] = t4; S.tau[5 * ne + e] = t5;
  S.sr[e] = s00; S.sr[ne + e] = s11; S.sr[2 * ne + e] = s22;
  S.sr[3 * ne + e] = s01; S.sr[4 * ne + e] = s12; S.sr[5 * ne + e] = s02;
  // the spin's diagonal stays zero (rows 0..2 are never written)
  S.rr[3 * ne + e] = w01; S.rr[4 * ne + e] = w12; S.rr[5 * ne + e] = w02;

  // element forces f = w * B^T sigma (3-D branch of calcElemForces)
  const double w = weight<NPE>();
#pragma unroll
  for (int a = 0; a < NPE; a++) {
    const double d0 = dH[0][a], d1 = dH[1][a], d2 = dH[2][a];
    // 0.0 + d * sigma * 1.0 of the reference is d * sigma (exact)
    double f0 = d0 * sg0, f1 = d1 * sg1, f2 = d2 * sg2;
    f0 += d1 * sg3 + d2 * sg5;
    f1 += d0 * sg3 + d2 * sg4;
    f2 += d1 * sg4 + d0 * sg5;
    S.fe[(3 * a) * ne + e] = f0 * w;
    S.fe[(3 * a + 1) * ne + e] = f1 * w;
    S.fe[(3 * a + 2) * ne + e] = f2 * w;
  }
}

// Tetrahedra with thermal coupling: the same quantities from the velocity
// gradient, (dN detJ) v / detJ with the velocities relative to node 0 (dN_0 is
// minus the sum of the others), in FMA form. The reference's node loop takes
// 156 FP64 instructions for the strain rate and spin, this 57, and its 4 x 4
// conduction matrix 16 divisions.
__global__ void __launch_bounds__(kElemThreads) k_fp64_tets_thermal(StepParams P, Fp64State S) {
  constexpr int NPE = 4;
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P.ne) return;
  const int64_t ne = P.ne;
  int32_t nid[NPE];
#pragma unroll
  for (int a = 0; a < NPE; a++) nid[a] = __ldg(&P.elnod[a * ne + e]);
  // A[k][m]: dN_(m+1)/dx_k detJ; node 0 has minus the row sums
  double A[3][3];
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int mm = 0; mm < 3; mm++) A[k][mm] = S.adj[(3 * k + mm) * ne + e];
  const double detJ = S.adj[9 * ne + e], vol = __ldg(&S.vol[e]);
  const int32_t mat_id = P.emat ? __ldg(&P.emat[e]) : 0;
  const MatDev &m = P.mats[mat_id];
  const double f = 1.0 / detJ, fh = 0.5 * f;
  double G[3][3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double v0 = __ldg(&S.vp[k * P.np + nid[0]]);
#pragma unroll
    for (int mm = 0; mm < 3; mm++) G[mm][k] = __ldg(&S.vp[k * P.np + nid[mm + 1]]) - v0;
  }
  auto AG = [&](int i, int k) {
    return fma(A[i][2], G[2][k], fma(A[i][1], G[1][k], A[i][0] * G[0][k]));
  };
  const double l10 = AG(1, 0), l01 = AG(0, 1), l21 = AG(2, 1), l12 = AG(1, 2), l20 = AG(2, 0),
               l02 = AG(0, 2);
  const double a00 = AG(0, 0), a11 = AG(1, 1), a22 = AG(2, 2);
  const double s01 = fh * (l10 + l01), w01 = fh * (l10 - l01);
  const double s12 = fh * (l21 + l12), w12 = fh * (l21 - l12);
  const double s02 = fh * (l20 + l02), w02 = fh * (l20 - l02);
  const long long step = P.st->step;
  const double c = thermal_strain_rate(P, S, m, nid, step);
  const double s00 = fma(a00, f, -c), s11 = fma(a11, f, -c), s22 = fma(a22, f, -c);
  const double p = element_pressure(P, S, m, e, nid, vol, P.stab_on ? a00 + a11 + a22 : 0.0);
  double SG[6], q_pl;
  stress_step<NPE, true>(P, S, m, mat_id, e, nid, s00, s11, s22, s01, s12, s02, w01, w12, w02, p,
                         vol, SG, q_pl);
  // forces f = w B^T sigma; node 0 balances the others
  const double w = weight<NPE>();
  const double Sk[3][3] = {{SG[0] * w, SG[3] * w, SG[5] * w},
                           {SG[3] * w, SG[1] * w, SG[4] * w},
                           {SG[5] * w, SG[4] * w, SG[2] * w}};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double sum = 0.0;
#pragma unroll
    for (int mm = 0; mm < 3; mm++) {
      const double v = fma(A[2][mm], Sk[2][k], fma(A[1][mm], Sk[1][k], A[0][mm] * Sk[0][k]));
      S.fe[(3 * (mm + 1) + k) * ne + e] = v;
      sum += v;
    }
    S.fe[k * ne + e] = -sum;
  }
  // conduction (K T)_i = (sum_d dN_i detJ sum_k dN_k detJ T_k) k_T / detJ w
  // through the temperature gradient, the temperatures relative to node 0
  const double T0 = S.T[nid[0]];
  double dT[3], gT[3], KT[NPE];
#pragma unroll
  for (int mm = 0; mm < 3; mm++) dT[mm] = S.T[nid[mm + 1]] - T0;
  const double kf = m.k_T * f * w;
#pragma unroll
  for (int i = 0; i < 3; i++)
    gT[i] = kf * fma(A[i][2], dT[2], fma(A[i][1], dT[1], A[i][0] * dT[0]));
#pragma unroll
  for (int mm = 0; mm < 3; mm++)
    KT[mm + 1] = fma(A[2][mm], gT[2], fma(A[1][mm], gT[1], A[0][mm] * gT[0]));
  KT[0] = -(KT[1] + KT[2] + KT[3]);
  store_temperature_rates(P, S, m, e, nid, step, KT, q_pl, vol);
}

// Hexahedra: the same quantities through the Walsh sums of the nodal values,
// with FMA. GB300 issues 2 FP64 instructions per SM and clock, so the FP64
// instruction count is the time: written out as the reference's loops over
// nodes and derivatives the element took 957 FP64 instructions. With
// X = 8 J the three derivative sums of the coordinates, A = adj(X) and
// D = det(X): volume D / 64, velocity gradient A G / D with G the velocity's
// derivative sums, nodal forces the synthesis of A^T sigma / 64, and the
// powers of two are exact.
template <bool TH>
__global__ void __launch_bounds__(kElemThreads) k_fp64_hexes(StepParams P, Fp64State S) {
  constexpr int NPE = 8;
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P.ne) return;
  const int64_t ne = P.ne;
  int32_t nid[NPE];
#pragma unroll
  for (int a = 0; a < NPE; a++) nid[a] = __ldg(&P.elnod[a * ne + e]);
  double A[3][3];
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int mm = 0; mm < 3; mm++) A[k][mm] = S.adj[(3 * k + mm) * ne + e];
  const double vol = __ldg(&S.vol[e]), D = vol * 64.0;
  const int32_t mat_id = P.emat ? __ldg(&P.emat[e]) : 0;
  const MatDev &m = P.mats[mat_id];
  double G[3][3];
  {
    // velocity sums; the hourglass forces depend on nothing else
    double ch = 0.0;
    if (P.hg_on) ch = P.hg_coef * pow_two_thirds(vol) * S.rho[e] * 0.25 * m.cs0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double v[8], o[8];
#pragma unroll
      for (int a = 0; a < 8; a++) v[a] = __ldg(&S.vp[k * P.np + nid[a]]);
      walsh8d(v, o);
      G[0][k] = o[1];
      G[1][k] = o[2];
      G[2][k] = o[3];
      if (P.hg_on) {
        double h[8];
        synth_hourglass(-(ch * o[4]), -(ch * o[5]), -(ch * o[6]), -(ch * o[7]), h);
#pragma unroll
        for (int a = 0; a < 8; a++) S.fhg[(3 * a + k) * ne + e] = h[a];
      }
    }
  }
  // strain rate and spin from L[i][k] = d v_k / d x_i = (A G)[i][k] / D
  const double f = 1.0 / D, fh = 0.5 * f;
  auto AG = [&](int i, int k) {
    return fma(A[i][2], G[2][k], fma(A[i][1], G[1][k], A[i][0] * G[0][k]));
  };
  double s00 = AG(0, 0) * f, s11 = AG(1, 1) * f, s22 = AG(2, 2) * f;
  const double l10 = AG(1, 0), l01 = AG(0, 1), l21 = AG(2, 1), l12 = AG(1, 2), l20 = AG(2, 0),
               l02 = AG(0, 2);
  const double s01 = fh * (l10 + l01), w01 = fh * (l10 - l01);
  const double s12 = fh * (l21 + l12), w12 = fh * (l21 - l12);
  const double s02 = fh * (l20 + l02), w02 = fh * (l20 - l02);
  // the divergence times detJ = D / 512
  const double div_v = P.stab_on ? (s00 + s11 + s22) * (D * (1.0 / 512.0)) : 0.0;
  const long long step = TH ? P.st->step : 0;
  if constexpr (TH) {
    const double c = thermal_strain_rate(P, S, m, nid, step);
    s00 = s00 - c;
    s11 = s11 - c;
    s22 = s22 - c;
  }
  const double p = element_pressure(P, S, m, e, nid, vol, div_v);

  double SG[6], q_pl;
  stress_step<NPE, TH>(P, S, m, mat_id, e, nid, s00, s11, s22, s01, s12, s02, w01, w12, w02, p, vol,
                       SG, q_pl);

  // forces: synthesis of A^T sigma / 64
  const double c64 = 1.0 / 64.0;
  const double sxx = SG[0] * c64, syy = SG[1] * c64, szz = SG[2] * c64, sxy = SG[3] * c64,
               syz = SG[4] * c64, sxz = SG[5] * c64;
  const double Sk[3][3] = {{sxx, sxy, sxz}, {sxy, syy, syz}, {sxz, syz, szz}};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double o[3], v[8];
#pragma unroll
    for (int mm = 0; mm < 3; mm++)
      o[mm] = fma(A[2][mm], Sk[2][k], fma(A[1][mm], Sk[1][k], A[0][mm] * Sk[0][k]));
    synth_linear(o[0], o[1], o[2], v);
#pragma unroll
    for (int a = 0; a < 8; a++) S.fe[(3 * a + k) * ne + e] = v[a];
  }
  if constexpr (TH) {
    // conduction in the same form: detJ grad T = A (sums of T) / 512,
    // (K T)_a = synthesis of A^T (detJ grad T) / 64 times k_T / detJ
    double tv[8], o[8], gT[3], KT[8];
#pragma unroll
    for (int a = 0; a < 8; a++) tv[a] = S.T[nid[a]];
    walsh8d(tv, o);
#pragma unroll
    for (int i = 0; i < 3; i++) gT[i] = fma(A[i][2], o[3], fma(A[i][1], o[2], A[i][0] * o[1]));
    const double kf = m.k_T * f * c64;
    double u[3];
#pragma unroll
    for (int mm = 0; mm < 3; mm++)
      u[mm] = kf * fma(A[2][mm], gT[2], fma(A[1][mm], gT[1], A[0][mm] * gT[0]));
    synth_linear(u[0], u[1], u[2], KT);
    store_temperature_rates(P, S, m, e, nid, step, KT, q_pl, vol);
  }
}

// ---------------------------------------------------------------------------
// Infinity or NaN, from the bits (no FP64 instruction).
__device__ __forceinline__ bool not_finite(double v) {
  return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}

// deterministic block sum (fixed shuffle tree, warps combined in order); a warp
// of zeros adds nothing and skips its five FP64 additions
__device__ __forceinline__ double block_sum(double v, double *sh) {
  if (__any_sync(0xffffffffu, __double_as_longlong(v) << 1 != 0)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += sh[i];
  }
  return t;
}

// Rigid triangle-mesh contact of the external nodes (Domain_d::CalcContactForces,
// Contact.C:31-334). tri_search finds a node's triangle: the first one, in
// order, that it penetrates (d < 0) with its projection inside. tri_contact
// forms its contact force.
//
// Does node x's plane distance and projection hit triangle j (Contact.C:58-120)?
__device__ __forceinline__ bool tri_hit(const StepParams &P, int32_t j, const double (&x)[3]) {
  const double n0 = P.tri_nrm[3 * j], n1 = P.tri_nrm[3 * j + 1], n2 = P.tri_nrm[3 * j + 2];
  const double dd = (n0 * x[0] + n1 * x[1] + n2 * x[2]) - P.tri_pp[j];
  if (!(dd < 0)) return false;
  const double Q[3] = {x[0] - n0 * dd, x[1] - n1 * dd, x[2] - n2 * dd};
  for (int l = 0; l < 3; l++) {
    const int nx = l + 1 > 2 ? 0 : l + 1;
    const double *a = &P.tri_x[3 * P.tri_el[3 * j + l]];
    const double *b = &P.tri_x[3 * P.tri_el[3 * j + nx]];
    const double e1[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
    const double e2[3] = {Q[0] - a[0], Q[1] - a[1], Q[2] - a[2]};
    const double c0 = e1[1] * e2[2] - e1[2] * e2[1];
    const double c1 = e1[2] * e2[0] - e1[0] * e2[2];
    const double c2 = e1[0] * e2[1] - e1[1] * e2[0];
    const double crit = c0 * n0 + c1 * n1 + c2 * n2;
    if (crit < 0.0) return false;
  }
  return true;
}

// The search of a block's nodes, all threads of the block taking part (act:
// this thread has an external node). The FP64 test costs about 70 FP64
// instructions a triangle, 16 cycles each on an SM of GB300, so the block
// first stages the triangles as FP32 copies relative to the die's first node
// (chunks of kTriChunk in shared memory) and rejects in FP32 what is certainly
// missed; what is left, mostly one or two triangles a node, takes the FP64
// test, in order, so the outcome is the FP64 search's. The margins: with R the
// largest relative coordinate involved, every FP32 quantity of length is
// within 2^-20 R and every product of two lengths within 2.4e-5 R^2 of its
// exact value; a distance is rejected above 1e-5 R, an edge test below
// -1e-4 R^2, and a comparison that involves an infinity or NaN rejects nothing.
// R is the die's extent, so an edge test's margin is 1e-4 R^2 / edge in distance: a
// tenth of an edge at 7 x 7 squares, several edges at 100 x 100, and the filter
// passes the more triangles the finer the die is. us a step of 72,000 tetrahedra,
// without and with it: 98 triangles 339 and 101, 2048 4197 and 432, 20,000 38,800
// and 5320, 180,000 349,000 and 115,000.
// 98 triangles over 13,671 nodes: 255 -> 85 us a step, the contact force and
// the die's motion included; with the kernel beside the element kernel and the
// FP64 tests of a warp taken together the whole step of 72,000 tetrahedra is
// 93 us, 393 before.
constexpr int kTriChunk = 64;
struct TriFilter {
  float n[3], pp, v[3][3], r;
};
__device__ __forceinline__ bool tri_miss(const TriFilter &f, const float (&xf)[3], float rx) {
  const float R = rx + f.r;
  const float d = f.n[0] * xf[0] + f.n[1] * xf[1] + f.n[2] * xf[2] - f.pp;
  if (d > 1e-5f * R) return true;
  const float q0 = xf[0] - f.n[0] * d, q1 = xf[1] - f.n[1] * d, q2 = xf[2] - f.n[2] * d;
  const float lim = -1e-4f * R * R;
  bool out = false;
#pragma unroll
  for (int l = 0; l < 3; l++) {
    const int nx = l == 2 ? 0 : l + 1;
    const float a0 = f.v[nx][0] - f.v[l][0], a1 = f.v[nx][1] - f.v[l][1],
                a2 = f.v[nx][2] - f.v[l][2];
    const float b0 = q0 - f.v[l][0], b1 = q1 - f.v[l][1], b2 = q2 - f.v[l][2];
    out |= (a1 * b2 - a2 * b1) * f.n[0] + (a2 * b0 - a0 * b2) * f.n[1] +
               (a0 * b1 - a1 * b0) * f.n[2] < lim;
  }
  return out;
}
__device__ __forceinline__ int32_t tri_search(const StepParams &P, bool act,
                                              const double (&x)[3], TriFilter *tf) {
  int32_t hit = -1;
  const double o0 = P.tri_x[0], o1 = P.tri_x[1], o2 = P.tri_x[2];
  float xf[3] = {0.f, 0.f, 0.f};
  if (act) {
    xf[0] = (float)(x[0] - o0);
    xf[1] = (float)(x[1] - o1);
    xf[2] = (float)(x[2] - o2);
  }
  const float rx = fmaxf(fmaxf(fabsf(xf[0]), fabsf(xf[1])), fabsf(xf[2]));
  for (int32_t j0 = 0; j0 < P.tri_ne; j0 += kTriChunk) {
    // also the barrier before a chunk is overwritten
    if (!__syncthreads_or(act && hit < 0)) break;
    const int m = min(kTriChunk, P.tri_ne - j0);
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const int32_t j = j0 + i;
      TriFilter f;
      const double n0 = P.tri_nrm[3 * j], n1 = P.tri_nrm[3 * j + 1], n2 = P.tri_nrm[3 * j + 2];
      f.n[0] = (float)n0;
      f.n[1] = (float)n1;
      f.n[2] = (float)n2;
      f.pp = (float)(P.tri_pp[j] - (n0 * o0 + n1 * o1 + n2 * o2));
      f.r = 0.f;
#pragma unroll
      for (int l = 0; l < 3; l++) {
        const double *a = &P.tri_x[3 * P.tri_el[3 * j + l]];
        f.v[l][0] = (float)(a[0] - o0);
        f.v[l][1] = (float)(a[1] - o1);
        f.v[l][2] = (float)(a[2] - o2);
#pragma unroll
        for (int k = 0; k < 3; k++) f.r = fmaxf(f.r, fabsf(f.v[l][k]));
      }
      tf[i] = f;
    }
    __syncthreads();
    // every lane advances to its next candidate, then all lanes test theirs
    // together: tested where each lane meets it, the FP64 test ran once for
    // every distinct triangle of a warp's nodes (contact kernel 75 us)
    bool live = act && hit < 0;
    int i = 0;
    while (__any_sync(0xffffffffu, live)) {
      if (live) {
        while (i < m && tri_miss(tf[i], xf, rx)) i++;
        live = i < m;
      }
      __syncwarp();
      if (live) {
        if (tri_hit(P, j0 + i, x)) {
          hit = j0 + i;
          live = false;
        }
        i++;
      }
    }
  }
  return hit;
}

// The contact force of an external node on its triangle j (-1: none): penalty
// normal force pf * min(E A / l, 0.2 m / dt^2) * d plus damping, then Coulomb
// friction from the accumulated tangential slip (static cap, else dynamic
// force along -v_t, slip reset). A node out of contact keeps its last contact
// force, as in the reference. Returns the normal-force magnitude when the
// triangle belongs to rigid body 0, the only body the reaction sums
// (Contact.C:229, :326-329), else 0.
__device__ __forceinline__ double tri_contact(const StepParams &P, const Fp64State &S, int64_t n,
                                              int32_t j, const double (&x)[3],
                                              const double (&v)[3], double m) {
  const int64_t np = P.np;
  double cfn = 0.0;
  if (j >= 0) {
    const double n0 = P.tri_nrm[3 * j], n1 = P.tri_nrm[3 * j + 1], n2 = P.tri_nrm[3 * j + 2];
    const double dd = (n0 * x[0] + n1 * x[1] + n2 * x[2]) - P.tri_pp[j];
    const double dt = P.dt;
    const double v_reln = v[0] * n0 + v[1] * n1 + v[2] * n2;
    const double kgeo = P.tri_E0 * P.node_area[n] / P.nodlen[n];
    const double kmass = 0.2 * m / (dt * dt);
    const double k = (kmass < kgeo) ? kmass : kgeo;
    const double omega = sqrt(k / m);
    const double ccrit = 2.0 * m * omega;
    const double F_damp = 0.2 * ccrit * v_reln;
    const double F_normal = P.tri_pf * k * dd;
    const double sc = -(F_normal + F_damp);
    double cf[3] = {n0 * sc, n1 * sc, n2 * sc};
    cfn = sqrt(cf[0] * cf[0] + cf[1] * cf[1] + cf[2] * cf[2]);
    // friction
    const double vn = v[0] * n0 + v[1] * n1 + v[2] * n2;
    const double vt[3] = {v[0] - n0 * vn, v[1] - n1 * vn, v[2] - n2 * vn};
    double ut[3] = {S.ut[n], S.ut[np + n], S.ut[2 * np + n]};
    const double du[3] = {vt[0] * dt, vt[1] * dt, vt[2] * dt};
    const double ua[3] = {ut[0] + du[0], ut[1] + du[1], ut[2] + du[2]};
    ut[0] += du[0];
    ut[1] += du[1];
    ut[2] += du[2];
    const double mk = -k;
    const double ft[3] = {ua[0] * mk, ua[1] * mk, ua[2] * mk};
    const double ft_mag = sqrt(ft[0] * ft[0] + ft[1] * ft[1] + ft[2] * ft[2]);
    const double cn = cf[0] * n0 + cf[1] * n1 + cf[2] * n2;
    const double Fn[3] = {n0 * cn, n1 * cn, n2 * cn};
    const double fn_norm = sqrt(Fn[0] * Fn[0] + Fn[1] * Fn[1] + Fn[2] * Fn[2]);
    double F[3];
    if (ft_mag <= P.tri_mu_s * fn_norm) {
      F[0] = ft[0];
      F[1] = ft[1];
      F[2] = ft[2];
    } else {
      const double md = -(P.tri_mu_d * fn_norm);
      const double vnorm = sqrt(vt[0] * vt[0] + vt[1] * vt[1] + vt[2] * vt[2]);
      const double inv = 1.0 / vnorm;
      F[0] = (vt[0] * md) * inv;
      F[1] = (vt[1] * md) * inv;
      F[2] = (vt[2] * md) * inv;
      ut[0] = ut[1] = ut[2] = 0.0;
    }
    S.ut[n] = ut[0];
    S.ut[np + n] = ut[1];
    S.ut[2 * np + n] = ut[2];
    cf[0] += F[0];
    cf[1] += F[1];
    cf[2] += F[2];
    if (P.tri_mid[j] != 0) cfn = 0.0;
    // heat from the die (Contact.C:309), kept after the contact ends
    if (P.thermal) S.qc[n] = P.tri_hc * P.node_area[n] * (P.tri_Tdie - S.T[n]);
    S.cf[n] = cf[0];
    S.cf[np + n] = cf[1];
    S.cf[2 * np + n] = cf[2];
  }
  return cfn;
}

// Triangle-mesh contact of the nodes of P.ext_list (external surface) and, by
// the last block, the die's motion to the next step. A kernel of its own that
// runs beside the element kernel (it needs only the nodal phase), off the
// step's chain of kernels; the node kernel picks up the forces (S.cf) and the
// reaction shares (S.cfn). A warp's FP64 instruction takes 64 cycles however
// many of its lanes are active, so the force of a node in contact (250 FP64
// instructions) and the die's motion (100) are some 12 us of latency. (8 bytes of
// spills.)
constexpr int kContactThreads = 128;
__global__ void __launch_bounds__(kContactThreads) k_fp64_contact(StepParams P, Fp64State S) {
  __shared__ TriFilter tf[kTriChunk];
  __shared__ bool am_last;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < P.n_ext;
  const double time = P.st->time;
  const int64_t n = act ? P.ext_list[i] : 0;
  double x[3];
#pragma unroll
  for (int k = 0; k < 3; k++) x[k] = act ? S.x[k * P.np + n] : 0.0;
  const int32_t hit = tri_search(P, act, x, tf);
  if (act) {
    const double v[3] = {S.vp[n], S.vp[P.np + n], S.vp[2 * P.np + n]};
    S.cfn[n] = tri_contact(P, S, n, hit, x, v, S.mass[n]);
  }
  // every block has read the die: the last one moves it
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    am_last = atomicAdd(&P.st->contact_blocks, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (am_last) {
    if (threadIdx.x == 0) P.st->contact_blocks = 0u;
    __threadfence();
    tri_move<false>(P, time);
  }
}

// nodes: assemblyForces (Matrices.C:42-87) as a gather over the node's
// element list, the non-finite clamp (Solver_explicit.C:777-785), plane
// contact (Contact.C:58-323), calcAccel (Mechanical.C:321-341), ImposeBCA,
// UpdateCorrectionAccVel (Domain_d.C:981-997), ImposeBCV,
// UpdateCorrectionPos (:1005-1025) and the next step's UpdatePrediction
// (:961-974) + ImposeBCV, which this kernel hands to the next step as vp.
// TRI: triangle-mesh dies.
template <int NPE, bool TRI>
__global__ void __launch_bounds__(kNodeThreads) k_fp64_nodes(StepParams P, Fp64State S) {
  __shared__ double sh[kNodeThreads / 32];
  __shared__ bool am_last;
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const double time = P.st->time;
  double r = 0.0;
  if (n < P.nn) {
    const int64_t np = P.np;
    const int32_t b = __ldg(&P.off[n]), c = __ldg(&P.off[n + 1]) - b;
    // the element forces, then the hourglass forces, each summed in list
    // order; eight entries at a time, so that a chunk's loads are in flight
    // together
    double fi[3] = {0.0, 0.0, 0.0}, fh[3] = {0.0, 0.0, 0.0}, sT = 0.0;
    for (int32_t k0 = 0; k0 < c; k0 += 8) {
      int64_t base[8];
      double g[8][3];
      if (P.thermal) {
        // the step's element-node temperature rates, in list order as well
        const double *cur = S.dte + (P.st->step & 1) * P.ne * NPE;
        double q[8];
#pragma unroll
        for (int j = 0; j < 8; j++) q[j] = (k0 + j < c) ? cur[__ldg(&P.slot[b + k0 + j])] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; j++) sT += q[j];
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int32_t sl = (k0 + j < c) ? __ldg(&P.slot[b + k0 + j]) : -1;
        base[j] = (sl >= 0) ? (int64_t)(sl % NPE) * 3 * P.ne + sl / NPE : -1;
      }
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int q = 0; q < 3; q++) g[j][q] = (base[j] >= 0) ? __ldg(&S.fe[base[j] + q * P.ne]) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int q = 0; q < 3; q++) fi[q] += g[j][q];
      if (P.hg_on) {
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
          for (int q = 0; q < 3; q++)
            g[j][q] = (base[j] >= 0) ? __ldg(&S.fhg[base[j] + q * P.ne]) : 0.0;
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
          for (int q = 0; q < 3; q++) fh[q] += g[j][q];
      }
    }
    if (P.hg_on) {
#pragma unroll
      for (int q = 0; q < 3; q++) fi[q] -= fh[q];
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (not_finite(fi[k])) {
        fi[k] = 0.0;
        atomicOr(&P.st->status, 1u);
        atomicMin(&P.st->first_bad_node, (long long)n);
      }
      S.fi[k * np + n] = fi[k];
    }
    const uint8_t fl = P.nflag[n];
    const double mass = S.mass[n];
    double x[3], vold[3], vp[3], pa[3], u[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      x[k] = S.x[k * np + n];
      vold[k] = S.v[k * np + n];
      vp[k] = S.vp[k * np + n];
      pa[k] = S.pa[k * np + n];
      u[k] = S.u[k * np + n];
    }
    double cf[3] = {0.0, 0.0, 0.0};
    if constexpr (TRI) {
      if (fl & NF_CONTACT) {   // from the contact kernel
#pragma unroll
        for (int k = 0; k < 3; k++) cf[k] = S.cf[k * np + n];
        r = S.cfn[n];
      }
    } else if (P.contact && (fl & NF_CONTACT)) {
      // rigid plane, outward normal (0, 0, -1), at z0 + vz * Time
      const double zd = P.c_z0 + P.c_vz * time;
      const double gap = zd - x[2];
      if (gap < 0) {
        // kcont = min(k_geometric, 0.2 m / dt^2) (Contact.C:190-193)
        const double kmass = 0.2 * mass / (P.dt * P.dt);
        const double k = (kmass < P.c_k) ? kmass : P.c_k;
        const double v_reln = vp[2] * -1.0;
        const double omega = sqrt(k / mass);
        const double ccrit = 2.0 * mass * omega;
        const double F_damp = 0.2 * ccrit * v_reln;
        const double F_normal = k * gap;
        const double cfz = -(F_normal + F_damp) * -1.0;
        cf[2] = cfz;
        r = fabs(cfz);
        double ut0 = S.ut[n] + vp[0] * P.dt;
        double ut1 = S.ut[np + n] + vp[1] * P.dt;
        double ftx = -k * ut0, fty = -k * ut1;
        const double ft_mag = sqrt(ftx * ftx + fty * fty);
        const double ft_max = P.c_mu * fabs(cfz);
        if (!(ft_mag <= ft_max)) {
          const double vt = sqrt(vp[0] * vp[0] + vp[1] * vp[1]);
          if (vt > 0.0) {
            ftx = -ft_max * vp[0] / vt;
            fty = -ft_max * vp[1] / vt;
          } else {
            ftx = fty = 0.0;
          }
          ut0 = ut1 = 0.0;
        }
        S.ut[n] = ut0;
        S.ut[np + n] = ut1;
        cf[0] += ftx;
        cf[1] += fty;
      }
      S.cf[n] = cf[0];
      S.cf[np + n] = cf[1];
      S.cf[2 * np + n] = cf[2];
    }
    if (!P.contact && (fl & NF_REACTION)) {
      const double fr = P.react_dim == 0 ? fi[0] : (P.react_dim == 1 ? fi[1] : fi[2]);
      if (P.rnode)
        P.rnode[n] = fr;  // summed per specimen by the reaction kernel
      else
        r = fr;
    }
    const uint32_t code = P.bc[n];
    const double *bv = &P.bcval[3 * (code >> 3)];
    const double dt = P.nspec_of ? P.spec_dt[P.nspec_of[n]] : P.dt;
    if constexpr (NPE == 8 || TRI) {
      // one reciprocal of the mass and the step's products formed once
      const double inv_m = 1.0 / mass;
      const double gdt = P.gamma * dt, pdt = (0.5 - P.beta) * dt, bdt2 = P.beta * dt * dt,
                   rdt = (1.0 - P.gamma) * dt;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const bool fixed = code & (1u << k);
        double a = (cf[k] - fi[k]) * inv_m;
        if (fixed) a = 0.0;
        a = P.fcorr * fma(-P.alpha, pa[k], a);
        double v = fma(gdt, a, vp[k]);
        if (fixed) v = bv[k];
        const double udt = fma(bdt2, a, dt * fma(pdt, pa[k], vold[k]));
        double vnext = fma(rdt, a, v);
        if (fixed) vnext = bv[k];
        S.x[k * np + n] = x[k] + udt;
        S.u[k * np + n] = u[k] + udt;
        S.v[k * np + n] = v;
        S.pa[k * np + n] = a;
        S.vp[k * np + n] = vnext;
      }
    } else {
      // the reference's operations in its order
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double a = (0.0 - fi[k]) / mass;
        if (P.contact) a += cf[k] / mass;
        if (code & (1u << k)) a = 0.0;
        a = P.fcorr * (a - P.alpha * pa[k]);
        double v = vp[k] + P.gamma * dt * a;
        if (code & (1u << k)) v = bv[k];
        double udt = dt * (vold[k] + (0.5 - P.beta) * dt * pa[k]);
        udt += P.beta * dt * dt * a;
        x[k] += udt;
        u[k] += udt;
        double vnext = v + (1.0 - P.gamma) * dt * a;
        if (code & (1u << k)) vnext = bv[k];
        S.x[k * np + n] = x[k];
        S.u[k * np + n] = u[k];
        S.v[k * np + n] = v;
        S.pa[k * np + n] = a;
        S.vp[k * np + n] = vnext;
      }
    }
    if (P.thermal) {
      // ThermalCalcs node part (Thermal.C:108-126): the gathered rates plus
      // the die heat over m cp of material 0
      S.T[n] = S.T[n] + (sT + S.qc[n] * 1.0 / (mass * P.cp0)) * P.dt;
    }
  }
  // reaction: block partial, then the last block to finish sums all partials
  // (each thread a fixed strided subset, then a fixed tree): deterministic.
  const double bs = block_sum(r, sh);
  if (threadIdx.x == 0) {
    P.partials[blockIdx.x] = bs;
    __threadfence();
    const unsigned prev = atomicAdd(&P.st->done_blocks, 1u);
    am_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (am_last) {
    __threadfence();
    double t = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x)
      t += ((volatile double *)P.partials)[i];
    const double tot = block_sum(t, sh);
    if (threadIdx.x == 0) {
      const long long s = P.st->step;
      if (s < P.hist_cap) P.hist[s] = tot;
      P.st->step = s + 1;
      P.st->time = time + P.dt;
      P.st->done_blocks = 0u;
    }
  }
}

// predictor for the first step of a run: vp = v + (1 - gamma) dt prev_a, BCs
__global__ void k_fp64_predict(StepParams P, Fp64State S) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.nn) return;
  const uint32_t code = P.bc[n];
  const double *bv = &P.bcval[3 * (code >> 3)];
  for (int k = 0; k < 3; k++) {
    const double dt = P.nspec_of ? P.spec_dt[P.nspec_of[n]] : P.dt;
    // rounded as the node kernel's predictor of the next step
    const double v0 = S.v[k * P.np + n], a0 = S.pa[k * P.np + n], c = (1.0 - P.gamma) * dt;
    double v = (P.npe == 8 || P.tri_on) ? fma(c, a0, v0) : v0 + c * a0;
    if (code & (1u << k)) v = bv[k];
    S.vp[k * P.np + n] = v;
  }
}

// calcElemDensity (Mechanical.C:295-319): rho = rho_0 * vol_0 / vol
__global__ void k_fp64_density(StepParams P, Fp64State S, const double *rho0) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P.ne) return;
  S.rho[e] = rho0[e] * S.vol0[e] / S.vol[e];
}

inline unsigned grid_for(int64_t n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

// Block size of the FP64 per-element and per-node kernels. GB300's FP64 rate
// per SM is low, so a small mesh is spread over more SMs with smaller blocks
// (down to one warp) until there are two blocks per SM; large meshes keep
// max_threads.
static int spread(int64_t n, int max_threads, int sms) {
  int t = max_threads;
  while (t > 32 && grid_for(n, t) < 2 * (int64_t)sms) t /= 2;
  return t;
}

int fp64_node_grid(int64_t nn, int sms) {
  return (int)grid_for(nn, spread(nn, kNodeThreads, sms));
}

void fp64_geometry(const StepParams &P, const Fp64State &S, cudaStream_t st, bool store_detj) {
  const int t = spread(P.ne, kElemThreads, P.sms);
  if (P.npe == 8)
    k_fp64_geometry<8><<<grid_for(P.ne, t), t, 0, st>>>(P, S, store_detj);
  else
    k_fp64_geometry<4><<<grid_for(P.ne, t), t, 0, st>>>(P, S, store_detj);
}

void fp64_nodal(const StepParams &P, const Fp64State &S, cudaStream_t st, int init_mode) {
  const int t = spread(P.nn, kNodeThreads, P.sms);
  if (P.npe == 8)
    k_fp64_nodal<8><<<grid_for(P.nn, t), t, 0, st>>>(P, S, init_mode);
  else
    k_fp64_nodal<4><<<grid_for(P.nn, t), t, 0, st>>>(P, S, init_mode);
}

void fp64_elements(const StepParams &P, const Fp64State &S, cudaStream_t st) {
  const int t = spread(P.ne, kElemThreads, P.sms);
  const unsigned g = (unsigned)grid_for(P.ne, t);
  if (P.npe == 8 && P.thermal)
    k_fp64_hexes<true><<<g, t, 0, st>>>(P, S);
  else if (P.npe == 8)
    k_fp64_hexes<false><<<g, t, 0, st>>>(P, S);
  else if (P.thermal)
    k_fp64_tets_thermal<<<g, t, 0, st>>>(P, S);
  else
    k_fp64_tets<<<g, t, 0, st>>>(P, S);
}

void fp64_nodes(const StepParams &P, const Fp64State &S, cudaStream_t st, int node_grid) {
  // node_grid = fp64_node_grid(P.nn, P.sms): blocks of the spread size
  const int t = spread(P.nn, kNodeThreads, P.sms);
  if (P.npe == 8 && P.tri_on)
    k_fp64_nodes<8, true><<<node_grid, t, 0, st>>>(P, S);
  else if (P.npe == 8)
    k_fp64_nodes<8, false><<<node_grid, t, 0, st>>>(P, S);
  else if (P.tri_on)
    k_fp64_nodes<4, true><<<node_grid, t, 0, st>>>(P, S);
  else
    k_fp64_nodes<4, false><<<node_grid, t, 0, st>>>(P, S);
}

void fp64_contact(const StepParams &P, const Fp64State &S, cudaStream_t st) {
  // at least one block: it moves the die
  const unsigned g = std::max(1u, grid_for(P.n_ext, kContactThreads));
  k_fp64_contact<<<g, kContactThreads, 0, st>>>(P, S);
}

void fp64_predict(const StepParams &P, const Fp64State &S, cudaStream_t st) {
  k_fp64_predict<<<grid_for(P.nn, kNodeThreads), kNodeThreads, 0, st>>>(P, S);
}

void fp64_density(const StepParams &P, const Fp64State &S, const double *rho0, cudaStream_t st) {
  k_fp64_density<<<grid_for(P.ne, kElemThreads), kElemThreads, 0, st>>>(P, S, rho0);
}

}  // namespace wf
