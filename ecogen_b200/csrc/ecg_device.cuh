// Device-side physics of the ECOGEN Cartesian FV step, in FP64.
//
// Every routine restates a reference routine (file:line relative to the ECOGEN
// tree) with the same operation order, so that results agree with the CPU code
// to the last bits except where a math function's result differs from glibc's by
// an ulp (epow, ecg_pow.cuh: in about 0.1 % of the calls, where glibc's pow is
// not correctly rounded; exp of the THINC reconstruction).  Divisions and square
// roots go through ndiv / dsqrt (ecg_ieee.cuh), which return the IEEE quotient and
// root bit for bit without a branch.  Kernels are built with --fmad=false so that
// no multiply-add is contracted, as in the reference's x86-64 SSE2 build.
//
// Compact state.  The reference keeps per phase (alpha, rho, p, T, e, c, Y) and per
// cell a mixture record (rho, p, u, e, E, cF, cWood).  After each full step every
// phase pressure equals the mixture-EOS pressure p clamped by that phase's EOS floor
// (FluxPUEq::correctionEnergy src/Models/PUEq/FluxPUEq.cpp:68-112 sets p_k = p then
// PhaseUEq::verifyAndCorrectPhase clamps it), and T, e, c, Y and the mixture record
// are pure functions of (alpha_k, rho_k, p_k, u).  So the state that defines a step is
// (alpha_k, rho_k)_k, p, u (DIM components) and E, and everything else is recomputed.
#pragma once
#include <cstdint>

#include "ecg_ieee.cuh"
#include "ecg_pow.cuh"
#include "ecg_types.h"

// Inlining of the two largest face routines (HLLC and the MUSCL side reconstruction).  Inlined, the
// fused pass holds one copy per axis and side; as calls, one copy each (smaller instruction
// footprint, call overhead).  Build-time choice, measured by the benchmark.
#ifndef ECG_HLLC_INLINE
#define ECG_HLLC_INLINE __forceinline__
#endif
#ifndef ECG_RECON_INLINE
#define ECG_RECON_INLINE __forceinline__
#endif

namespace ecg {

// std::max / std::min with libstdc++'s argument order (NaN behaviour included)
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

// ----------------------------------------------------------------------------------------- EOS
// src/Eos/EosIG.cpp:64-257, src/Eos/EosSG.cpp:66-257, src/Eos/EosNASG.cpp:68-280

__device__ __forceinline__ double eos_T(const EosParams& q, double eps, double rho, double p) {
  if (q.type == ECG_EOS_IG) return ndiv(ndiv(cdiv(p, q.gm1, q.ig), dmax(rho, eps)), q.cv);
  if (q.type == ECG_EOS_SG) return ndiv(ndiv(cdiv(p + q.pinf, q.gm1, q.ig), dmax(rho, eps)), q.cv);
  return ndiv(ndiv(cdiv((p + q.pinf) * dmax(1. - rho * q.b, eps), q.gm1, q.ig), q.cv), dmax(rho, eps));
}

__device__ __forceinline__ double eos_e(const EosParams& q, double eps, double rho, double p) {
  if (q.type == ECG_EOS_IG) return ndiv(cdiv(p, q.gm1, q.ig), dmax(rho, eps)) + q.eref;
  if (q.type == ECG_EOS_SG) return ndiv(cdiv(p + q.gpinf, q.gm1, q.ig), dmax(rho, eps)) + q.eref;
  return ndiv(cdiv((p + q.gpinf) * dmax(1. - rho * q.b, eps), q.gm1, q.ig), dmax(rho, eps)) + q.eref;
}

__device__ __forceinline__ double eos_p(const EosParams& q, double eps, double rho, double e) {
  if (q.type == ECG_EOS_IG) return q.gm1 * rho * (e - q.eref);
  if (q.type == ECG_EOS_SG) return q.gm1 * rho * (e - q.eref) - q.gpinf;
  return (ndiv(rho * q.gm1 * (e - q.eref), dmax(1. - rho * q.b, eps)) - q.gpinf);
}

// eos_e and eos_c of a density that phase_fix_ar has clamped: rho >= 1e-15 >= eps (or NaN), so the floor
// dmax(rho, eps) of the ideal and stiffened gas is the density itself.
__device__ __forceinline__ double eos_e_clamped(const EosParams& q, double eps, double rho, double p) {
  if (q.type == ECG_EOS_IG) return ndiv(cdiv(p, q.gm1, q.ig), rho) + q.eref;
  if (q.type == ECG_EOS_SG) return ndiv(cdiv(p + q.gpinf, q.gm1, q.ig), rho) + q.eref;
  return eos_e(q, eps, rho, p);
}

__device__ __forceinline__ double eos_c(const EosParams& q, double eps, double rho, double p) {
  if (q.type == ECG_EOS_IG) return dsqrt(ndiv(q.gamma * p, dmax(rho, eps)));
  if (q.type == ECG_EOS_SG) return dsqrt(ndiv(q.gamma * (p + q.pinf), dmax(rho, eps)));
  return dsqrt(ndiv(q.gamma * (p + q.pinf), dmax(rho * (1. - rho * q.b), eps)));
}

__device__ __forceinline__ double eos_c_clamped(const EosParams& q, double eps, double rho, double p) {
  if (q.type == ECG_EOS_IG) return dsqrt(ndiv(q.gamma * p, rho));
  if (q.type == ECG_EOS_SG) return dsqrt(ndiv(q.gamma * (p + q.pinf), rho));
  return eos_c(q, eps, rho, p);
}

__device__ __forceinline__ double nonzero(double a, double eps) {  // Tools::returnNonZeroValue src/Tools.cpp:134
  if (a > eps || a < -eps) return a;
  int sg = (0. < a) - (a < 0.);
  return sg * eps;
}

template <bool CLAMPED>
__device__ __forceinline__ double eos_p_isentropic(const EosParams& q, double eps, double p0, double rho0,
                                                   double rho1) {
  const double ratio = ndiv(rho1, CLAMPED ? rho0 : dmax(rho0, eps));
  if (q.type == ECG_EOS_IG) return p0 * epow(ratio, q.gamma);
  if (q.type == ECG_EOS_SG) return (p0 + q.pinf) * epow(ratio, q.gamma) - q.pinf;
  return (p0 + q.pinf) * epow(ratio, q.gamma) * epow(ndiv(1. - rho0 * q.b, 1. - rho1 * q.b), q.gamma) -
         q.pinf;
}

__device__ __forceinline__ double eos_rho_pfinal(const EosParams& q, double eps, double p0, double rho0, double p1,
                                                 double* drhodp) {
  double num, denom, rho1;
  if (q.type == ECG_EOS_IG) {
    num = q.gamma * p1;
    denom = num + p0 - p1;
    rho1 = ndiv(rho0 * num, dmax(denom, eps));
    *drhodp = ndiv(rho0 * q.gamma * p0, dmax(denom * denom, eps));
    return rho1;
  }
  if (q.type == ECG_EOS_SG) {
    num = q.gamma * (p1 + q.pinf);
    denom = num + p0 - p1;
    rho1 = ndiv(rho0 * num, nonzero(denom, eps));
    *drhodp = ndiv(rho0 * q.gamma * (p0 + q.pinf), dmax(denom * denom, eps));
    return rho1;
  }
  num = q.gamma * (p1 + q.pinf);
  denom = num + p0 - p1 + q.b * rho0 * (p1 - p0);
  rho1 = ndiv(rho0 * num, nonzero(denom, eps));
  *drhodp = ndiv(rho0 * q.gamma * (p0 + q.pinf - q.b * rho0 * (p0 + q.pinf)), nonzero(denom * denom, eps));
  return rho1;
}

// verifyAndModifyPressure (EosIG.cpp:250, EosSG.cpp:252, EosNASG.cpp:268)
__device__ __forceinline__ double eos_fix_p(const EosParams& q, double p) { return (p < q.pfloor) ? q.pfloor : p; }

__device__ __forceinline__ void eos_rho_max(const EosParams& q, double& rho) {  // verifyAndCorrectDensityMax(density)
  if (q.type == ECG_EOS_NASG && rho > ndiv(1., q.b) - 1.) rho = ndiv(1., q.b) - 1.;
}

// ------------------------------------------------------------------------------ model parameters

template <int NP>
struct Model {
  EosParams eos[NP];
  double eps;  // epsilonAlphaNull: 1e-15 with alphaNull, else 0 (src/Eos/Eos.cpp:88-97)
};

// Kernel configuration known at compile time ("fast" kernels): the type of phase k in bits
// 2k..2k+1 (ECG_EOS_IG 0, SG 1, NASG 2) and, in bits 8 and up, one more than a limiter used for all
// four limiter slots (0: limiters read at run time).  EOS_DYNAMIC marks the generic kernels.  With
// known types and limiter every EOS and limiter branch folds away (the arithmetic is unchanged),
// which shrinks the fused kernels' code.
constexpr int EOS_DYNAMIC = -1;
template <int NP>
__host__ __device__ constexpr int eos_types_code(int t0, int t1, int t2 = 0) {
  return NP == 2 ? (t0 | (t1 << 2)) : (t0 | (t1 << 2) | (t2 << 4));
}
__host__ __device__ constexpr int fast_code(int types, int limiter) { return types | ((limiter + 1) << 8); }
__host__ __device__ constexpr int code_limiter(int code) { return code == EOS_DYNAMIC ? -1 : (code >> 8) - 1; }
template <int NP, int TYPES>
__device__ __forceinline__ Model<NP> specialize_eos(const Model<NP>& M0) {
  Model<NP> M = M0;
  if (TYPES != EOS_DYNAMIC) {
#pragma unroll
    for (int k = 0; k < NP; k++) M.eos[k].type = (TYPES >> (2 * k)) & 3;
  }
  return M;
}

// PhaseUEq::verifyAndCorrectPhase src/Models/UEq/PhaseUEq.cpp:348 (alpha / density clamps)
__device__ __forceinline__ void phase_fix_ar(double eps, double& a, double& r) {
  if (eps > 1.e-20) {
    if (a < 0.) a = 0.;
    if (a > 1.) a = 1.;
    if (r <= 1.e-15) r = 1.e-15;
  } else {
    if (a < 1e-15) a = 1e-14;
    if (a > 1. - 1e-15) a = 1. - 1e-14;
    if (r < 1.e-15) r = 1.e-14;
  }
}

// Thermodynamic closure of one side of a face or of a cell: what fulfillState computes
// (ModUEq::fulfillState src/Models/UEq/ModUEq.cpp:99 -> PhaseUEq::extendedCalculusPhase :97,
// MixUEq::computeMixtureVariables src/Models/UEq/MixUEq.cpp:136).
// The phase internal energies e_k and the mixture energy sum_k Y_k e_k are needed only on the side
// the HLLC solution is sampled from, so hllc() evaluates them once the side is known
// (hllc_side_energy); the values are the ones fulfillState would have produced.
template <int NP>
struct Thermo {
  double a[NP], r[NP], p[NP], Y[NP];
  double rho, pm, cF;
};

// CLAMPED: the densities have been through phase_fix_ar (a reconstructed side).
template <int NP, bool CLAMPED = false>
__device__ __forceinline__ void fulfill(const Model<NP>& M, Thermo<NP>& t) {
  double c[NP];
#pragma unroll
  for (int k = 0; k < NP; k++)
    c[k] = CLAMPED ? eos_c_clamped(M.eos[k], M.eps, t.r[k], t.p[k]) : eos_c(M.eos[k], M.eps, t.r[k], t.p[k]);
  t.rho = 0.;
  t.pm = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    t.rho += t.a[k] * t.r[k];
    t.pm += t.a[k] * t.p[k];
  }
  double cF = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    t.Y[k] = ndiv(t.a[k] * t.r[k], dmax(t.rho, M.eps));
    cF += t.Y[k] * c[k] * c[k];
  }
  t.cF = dsqrt(cF);
}

// PhaseUEq::extendedCalculusPhase energies and MixUEq::computeMixtureVariables' e = sum_k Y_k e_k.
template <int NP, bool CLAMPED = false>
__device__ __forceinline__ double side_energy(const Model<NP>& M, const Thermo<NP>& t, double e[NP]) {
  double em = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    e[k] = CLAMPED ? eos_e_clamped(M.eos[k], M.eps, t.r[k], t.p[k]) : eos_e(M.eos[k], M.eps, t.r[k], t.p[k]);
    em += t.Y[k] * e[k];
  }
  return em;
}

// Face-frame projection of a Cartesian face (src/Maths/Coord.cpp:133-151 with the frames of
// src/Meshes/MeshCartesian.cpp:281-557).  axis 0/1/2; neg = true for the Xm/Ym/Zm boundary frames.
__device__ __forceinline__ void to_local(int axis, bool neg, const double u[3], double l[3]) {
  if (axis == 0) {
    if (!neg) { l[0] = u[0]; l[1] = u[1]; l[2] = u[2]; }
    else { l[0] = -u[0]; l[1] = -u[1]; l[2] = u[2]; }
  } else if (axis == 1) {
    if (!neg) { l[0] = u[1]; l[1] = -u[0]; l[2] = u[2]; }
    else { l[0] = -u[1]; l[1] = u[0]; l[2] = u[2]; }
  } else {
    if (!neg) { l[0] = u[2]; l[1] = u[0]; l[2] = u[1]; }
    else { l[0] = -u[2]; l[1] = -u[0]; l[2] = u[1]; }
  }
}
__device__ __forceinline__ void to_global(int axis, bool neg, const double f[3], double g[3]) {
  if (axis == 0) {
    if (!neg) { g[0] = f[0]; g[1] = f[1]; g[2] = f[2]; }
    else { g[0] = -f[0]; g[1] = -f[1]; g[2] = f[2]; }
  } else if (axis == 1) {
    if (!neg) { g[0] = -f[1]; g[1] = f[0]; g[2] = f[2]; }
    else { g[0] = f[1]; g[1] = -f[0]; g[2] = f[2]; }
  } else {
    if (!neg) { g[0] = f[1]; g[1] = f[2]; g[2] = f[0]; }
    else { g[0] = -f[1]; g[1] = f[2]; g[2] = -f[0]; }
  }
}

// The time-step restriction of the faces a thread solves, min lCFL / |s| over the waves faster than 1e-3,
// carried as a value to be maximised: the fastest |s| itself on a uniform mesh, where every cell has the
// same lCFL and a correctly rounded quotient falls monotonically with its divisor, so that the minimum of
// the quotients is the quotient by the maximum (one division per block in place of two per face); minus
// the smallest lCFL / |s| on a stretched mesh.  A NaN speed is ignored, as in the minimum.
__device__ __forceinline__ double wave_none(bool stretched) { return stretched ? -1.e10 : 0.; }
__device__ __forceinline__ void wave_add(double& w, bool stretched, double s, double lcfl) {
  if (!stretched) w = dmax(w, fabs(s));
  else if (fabs(s) > 1.e-3) w = dmax(w, -ndiv(1. * lcfl, fabs(s)));
}
__device__ __forceinline__ double wave_dtmax(double w, bool stretched, double lcfl) {
  if (stretched) return -w;
  return (w > 1.e-3) ? dmin(1.e10, ndiv(1. * lcfl, w)) : 1.e10;
}

// Face flux of the Kapila / UEq system, in the absolute frame.
template <int NP>
struct Flux {
  double a[NP], m[NP], en[NP];
  double mom[3];
  double E;
  double sM, uStar;
};

// HLLC: ModUEq::solveRiemannIntern src/Models/UEq/ModUEq.cpp:113-267.  L and R carry local-frame
// velocities ul/ur (normal first).  wmax collects the wave speeds (wave_add).  CLAMPED: see fulfill.
template <int NP, bool CLAMPED = false>
__device__ ECG_HLLC_INLINE void hllc(const Model<NP>& M, const Thermo<NP>& L, const double ul[3],
                                     const Thermo<NP>& R, const double ur[3], bool stretched, double dxL,
                                     double dxR, double& wmax, double Fn[3], Flux<NP>& F) {
  double uL = ul[0], cL = L.cF, pL = L.pm, rhoL = L.rho;
  double uR = ur[0], cR = R.cF, pR = R.pm, rhoR = R.rho;
  double sL = dmin(uL - cL, uR - cR);
  double sR = dmax(uR + cR, uL + cL);
  wave_add(wmax, stretched, sL, dxL);
  wave_add(wmax, stretched, sR, dxR);
  double mL = rhoL * (sL - uL), mR = rhoR * (sR - uR);
  double sM = ndiv(pR - pL + mL * uL - mR * uR, mL - mR);
  if (fabs(sM) < 1.e-8) sM = 0.;
  F.sM = sM;
  if (sL >= 0. || sR <= 0.) {
    const bool left = (sL >= 0.);
    const Thermo<NP>& S = left ? L : R;
    const double* us = left ? ul : ur;
    double un = us[0], rhoS = S.rho, pS = S.pm;
    double e[NP];
    const double em = side_energy<NP, CLAMPED>(M, S, e);
#pragma unroll
    for (int k = 0; k < NP; k++) {
      F.a[k] = S.a[k] * sM;
      F.m[k] = S.a[k] * S.r[k] * un;
      F.en[k] = S.a[k] * S.r[k] * e[k] * un;
    }
    double Et = em + 0.5 * (us[0] * us[0] + us[1] * us[1] + us[2] * us[2]);
    Fn[0] = rhoS * un * un + pS;
    Fn[1] = rhoS * us[1] * un;
    Fn[2] = rhoS * us[2] * un;
    F.E = (rhoS * Et + pS) * un;
    F.uStar = un;
  } else {
    const bool left = (sM >= 0.);
    const Thermo<NP>& S = left ? L : R;
    const double* us = left ? ul : ur;
    double sK = left ? sL : sR;
    double mK = left ? mL : mR;
    double uK = us[0], pK = S.pm;
    double e[NP];
    const double em = side_energy<NP, CLAMPED>(M, S, e);
    double Et = em + 0.5 * (us[0] * us[0] + us[1] * us[1] + us[2] * us[2]);
    double rhoStar = ndiv(mK, sK - sM);
    double EStar = Et + (sM - uK) * (sM + ndiv(pK, mK));
    double pStar = mK * (sM - uK) + pK;
#pragma unroll
    for (int k = 0; k < NP; k++) {
      double mk = S.r[k] * (sK - uK);
      double rks = ndiv(mk, sK - sM);
      eos_rho_max(M.eos[k], rks);
      double pks = eos_p_isentropic<CLAMPED>(M.eos[k], M.eps, S.p[k], S.r[k], rks);
      double eks = eos_e(M.eos[k], M.eps, rks, pks);
      F.a[k] = S.a[k] * sM;
      F.m[k] = S.a[k] * rks * sM;
      F.en[k] = S.a[k] * rks * eks * sM;
    }
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * us[1] * sM;
    Fn[2] = rhoStar * us[2] * sM;
    F.E = (rhoStar * EStar + pStar) * sM;
    F.uStar = sM;
  }
}

// fulfill and hllc of an internal face, for operands in their ordinary range: the same quotients and roots from
// shorter sequences.  A division's reciprocal serves every quotient by that divisor and, scaled, by the star
// densities (1/rho_k* = (1/rho_k)(s_K - s_M)/(s_K - u_K) to a few ulps, which qdiv's correction allows), and no
// quotient or root tests for zero, infinite or NaN operands: hllc_quick returns false when a phase is NASG, a
// density is at its floor or a result is NaN, as every special operand makes it, and the caller then solves the
// face by fulfill and hllc.  Measured with the same bits (one B200, mid-run states): face kernels 2D 2048^2
// 0.311 / 0.291 -> 0.303 / 0.286 ms, 3D 256^3 1.91 / 1.64 / 1.64 -> 1.79 / 1.61 / 1.62 ms (X faces with the
// domain sides solved beside the others), THINC 1000 x 601 0.099 / 0.094 -> 0.073 / 0.066 ms (the general face
// and its sides out of line); 4096 tubes 3.28 -> 3.05 ms per step.  LOW: the densities and pressures may lie below the
// floors (sides not clamped by phase_fix_ar and eos_fix_p).
template <int NP>
__device__ __forceinline__ void fulfill_quick(const Model<NP>& M, Thermo<NP>& t) {
  double c[NP];
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const EosParams& q = M.eos[k];
    const double pi = q.type == ECG_EOS_IG ? 0. : q.pinf;
    c[k] = qsqrt(qdiv(q.gamma * (t.p[k] + pi), t.r[k], nrcp(t.r[k])));
  }
  t.rho = 0.;
  t.pm = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    t.rho += t.a[k] * t.r[k];
    t.pm += t.a[k] * t.p[k];
  }
  const double y = nrcp(t.rho);
  double cF = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    t.Y[k] = qdiv(t.a[k] * t.r[k], t.rho, y);
    cF += t.Y[k] * c[k] * c[k];
  }
  t.cF = qsqrt(cF);
}

template <int NP, bool LOW>
__device__ __forceinline__ bool hllc_quick(const Model<NP>& M, Thermo<NP>& L, const double ul[3], Thermo<NP>& R,
                                           const double ur[3], bool stretched, double dxL, double dxR, double& wmax,
                                           double Fn[3], Flux<NP>& F, bool ok = true) {
#pragma unroll
  for (int k = 0; k < NP; k++) {
    ok = ok && M.eos[k].type != ECG_EOS_NASG;
    if (LOW)
      ok = ok && L.r[k] >= 1.e-15 && R.r[k] >= 1.e-15 && L.p[k] >= M.eos[k].pfloor && R.p[k] >= M.eos[k].pfloor;
  }
  fulfill_quick<NP>(M, L);
  fulfill_quick<NP>(M, R);
  ok = ok && L.rho > 1.e-15 && R.rho > 1.e-15;
  const double uL = ul[0], cL = L.cF, pL = L.pm, rhoL = L.rho;
  const double uR = ur[0], cR = R.cF, pR = R.pm, rhoR = R.rho;
  const double sL = dmin(uL - cL, uR - cR), sR = dmax(uR + cR, uL + cL);
  const double mL = rhoL * (sL - uL), mR = rhoR * (sR - uR), dm = mL - mR;
  double sM = qdiv(pR - pL + mL * uL - mR * uR, dm, nrcp(dm));
  if (fabs(sM) < 1.e-8) sM = 0.;
  F.sM = sM;
  const bool plain = sL >= 0. || sR <= 0.;
  const bool left = plain ? (sL >= 0.) : (sM >= 0.);
  const Thermo<NP>& S = left ? L : R;
  const double* us = left ? ul : ur;
  const double un = us[0], rhoS = S.rho, pS = S.pm;
  double e[NP], yr[NP], em = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const EosParams& q = M.eos[k];
    const double gp = q.type == ECG_EOS_IG ? 0. : q.gpinf;
    yr[k] = nrcp(S.r[k]);
    e[k] = qdiv(qdiv(S.p[k] + gp, q.gm1, q.ig), S.r[k], yr[k]) + q.eref;
    em += S.Y[k] * e[k];
  }
  const double Et = em + 0.5 * (us[0] * us[0] + us[1] * us[1] + us[2] * us[2]);
  if (plain) {
#pragma unroll
    for (int k = 0; k < NP; k++) {
      F.a[k] = S.a[k] * sM;
      F.m[k] = S.a[k] * S.r[k] * un;
      F.en[k] = S.a[k] * S.r[k] * e[k] * un;
    }
    Fn[0] = rhoS * un * un + pS;
    Fn[1] = rhoS * us[1] * un;
    Fn[2] = rhoS * us[2] * un;
    F.E = (rhoS * Et + pS) * un;
    F.uStar = un;
  } else {
    const double sK = left ? sL : sR, mK = left ? mL : mR;
    const double dK = sK - un, d = sK - sM, y = nrcp(d);
    const double yd = d * nrcp(dK);  // (s_K - s_M) / (s_K - u_K)
    const double rhoStar = qdiv(mK, d, y);
    const double EStar = Et + (sM - un) * (sM + qdiv(pS, mK, nrcp(mK)));
    const double pStar = mK * (sM - un) + pS;
#pragma unroll
    for (int k = 0; k < NP; k++) {
      const EosParams& q = M.eos[k];
      const double pi = q.type == ECG_EOS_IG ? 0. : q.pinf, gp = q.type == ECG_EOS_IG ? 0. : q.gpinf;
      const double rks = qdiv(S.r[k] * dK, d, y);
      ok = ok && rks > 1.e-15;
      const double pks = (S.p[k] + pi) * epow(qdiv(rks, S.r[k], yr[k]), q.gamma) - pi;
      const double eks = qdiv(qdiv(pks + gp, q.gm1, q.ig), rks, yr[k] * yd) + q.eref;
      F.a[k] = S.a[k] * sM;
      F.m[k] = S.a[k] * rks * sM;
      F.en[k] = S.a[k] * rks * eks * sM;
    }
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * us[1] * sM;
    Fn[2] = rhoStar * us[2] * sM;
    F.E = (rhoStar * EStar + pStar) * sM;
    F.uStar = sM;
  }
  double t = F.E + (cL + cR) + F.sM;
#pragma unroll
  for (int k = 0; k < NP; k++) t += F.en[k];
  if (!(ok && t == t)) return false;
  wave_add(wmax, stretched, sL, dxL);
  wave_add(wmax, stretched, sR, dxR);
  return true;
}

// Limiters src/Order2/Limiter{Minmod,VanLeer,VanAlbada,SuperBee,MC,THINC}.cpp:43-55
__device__ __forceinline__ double limiter(int kind, double s1, double s2) {
  double slope = 0., prod = s1 * s2;
  switch (kind) {
    case ECG_LIM_MINMOD:
    case ECG_LIM_THINC:
      if (prod > 1e-9) {
        slope = dmin(fabs(s1), fabs(s2));
        if (s1 < 0) slope = -slope;
      }
      return slope;
    case ECG_LIM_VANLEER: {
      double sum = s1 + s2;
      if ((fabs(sum) > 1e-6) && (prod > 1e-6)) slope = ndiv(2. * prod, sum);
      return slope;
    }
    case ECG_LIM_VANALBADA: {
      double sum = s1 + s2;
      if ((fabs(s1) > 1e-6) && (fabs(s2) > 1e-6) && (fabs(sum) > 1e-6) && (prod > 1e-6))
        slope = ndiv(prod * sum, s1 * s1 + s2 * s2);
      return slope;
    }
    case ECG_LIM_SUPERBEE:
      if (prod > 1e-6) slope = dmax(dmin(2. * fabs(s1), fabs(s2)), dmin(fabs(s1), 2. * fabs(s2)));
      if (s1 < 0.) slope = -slope;
      return slope;
    case ECG_LIM_MC:
      if (prod > 1e-9) {
        slope = dmin(2. * fabs(s1), 2. * fabs(s2));
        slope = dmin(slope, 0.5 * (fabs(s1) + fabs(s2)));
      }
      if (s1 < 0.) slope = -slope;
      return slope;
    default:
      return 0.;
  }
}

// ------------------------------------------------------------------------ relaxation (pressure)

struct RelaxStats {
  int iters;      // Newton evaluations of this cell (0 if skipped)
  bool fallback;  // reached 100 iterations -> interface pressure
  bool seeded;    // a learned seed was used
  bool rejected;  // the learned seed was rejected (plain start used)
};

// A Newton state after `it` evaluations at the iterates up to ps (RelaxationP::NewtonRaphson
// src/Relaxations/RelaxationP.cpp:43-68): f = sum_k alpha_k rho_k / rho_k*(ps) - 1, its derivative df, and an
// approximate reciprocal ydf of df (NaN: none).
struct NewtonState {
  double ps, f, df;
  int it;
  double ydf;
};

// One evaluation, term by term (the general form).
template <int NP>
__device__ __forceinline__ void pinf_eval_general(const Model<NP>& M, const double a[NP], const double r[NP],
                                                      NewtonState& s, const double p[NP], double aS[NP],
                                                      double rS[NP]) {
  double drhodp = 0.;
  s.f = -1.;
  s.df = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    rS[k] = eos_rho_pfinal(M.eos[k], M.eps, p[k], r[k], s.ps, &drhodp);
    aS[k] = ndiv(a[k] * r[k], rS[k]);
    const double dalpha = ndiv(a[k] * r[k] * drhodp, rS[k] * rS[k]);
    s.f += aS[k];
    s.df -= dalpha;
  }
  s.ydf = __longlong_as_double(0x7ff8000000000000ll);
}

// One evaluation at s.ps, after verifyAndModifyPressure of every phase.
//
// The iteration is a serial chain, up to 60 evaluations long in the cells of a contact, and those cells set the
// time of a small mesh's step.  Term by term it holds three dependent divisions, each a reciprocal sequence
// (an approximation and two Newton steps) and a correction.  The quotients and their order are the same here,
// but the reciprocals come from values at hand before the exact divisors: with rho* = rho num / denom,
// 1/denom and 1/(rho num) start side by side, 1/rho* is denom (1/(rho num)), the squares' reciprocals are the
// reciprocals' squares, and 1/df is taken from the derivative assembled from them, while f and df themselves
// are still being rounded.  A quotient corrected with a reciprocal of a few ulps' error is RN(a / b) unless
// a / b lies within 2^-47 ulp of a midpoint (the residual is exact, the correction a product of two errors).
// Measured with the same bits (one B200, mid-run states, per step): tube of 1000 cells, whose contact cells need
// 55 evaluations, 25.4 -> 23.1 us; cell kernels of 191 x 103 cells 32 / 34 -> 23 / 23 us, of 2048^2 0.41 / 0.43
// -> 0.36 / 0.37 ms, of 256^3 (three phases, at most 6 evaluations) 2.36 / 2.38 -> 2.24 / 2.27 ms.  With the
// general form as a branch inside the loop the three-phase cell kernel spilled 192 bytes and took 2.46 ms.
// Returns false where the general form has to run: for NASG phases, and where a divisor lies near its floor or
// an operand is zero, infinite or NaN (f or df is NaN then), or where the terms of df cancel.
template <int NP>
__device__ __forceinline__ bool pinf_quick(const Model<NP>& M, const double a[NP], const double r[NP], NewtonState& s,
                                          const double p[NP], double aS[NP], double rS[NP]) {
#pragma unroll
  for (int k = 0; k < NP; k++) s.ps = eos_fix_p(M.eos[k], s.ps);
  const double ps = s.ps;
  double f = -1., df = 0., dfa = 0.;
  bool plain = true;
  const double low = M.eps > 0. ? 1.e-7 : 1.e-140;  // above it eos_rho_pfinal's floors of denom and denom^2 do nothing
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const EosParams& q = M.eos[k];
    plain = plain && q.type != ECG_EOS_NASG;
    const double pi = q.type == ECG_EOS_IG ? 0. : q.pinf;
    const double num = q.type == ECG_EOS_IG ? q.gamma * ps : q.gamma * (ps + pi);
    const double denom = num + p[k] - ps;
    plain = plain && denom > low;
    const double rn = r[k] * num, d2 = denom * denom, ar = a[k] * r[k];
    const double c = q.type == ECG_EOS_IG ? r[k] * q.gamma * p[k] : r[k] * q.gamma * (p[k] + pi);
    const double yd = nrcp(denom), yn = nrcp(rn);
    const double yr = denom * yn, yd2 = yd * yd, yr2 = yr * yr;
    dfa -= (ar * c) * (yd2 * yr2);
    const double rho = qdiv(rn, denom, yd);
    const double drhodp = qdiv(c, d2, yd2);
    const double as = qdiv(ar, rho, yr);
    const double dalpha = qdiv(ar * drhodp, rho * rho, yr2);
    rS[k] = rho;
    aS[k] = as;
    f += as;
    df -= dalpha;
  }
  s.f = f;
  s.df = df;
  s.ydf = nrcp(dfa);
  // df sums terms of one sign (densities, volume fractions and p + pInf are positive), so 1/dfa is 1/df to a few
  // ulps; checked all the same
  return plain && f == f && fabs(fma(df, s.ydf, -1.)) < 1.e-12;
}

// One evaluation in either form (the seeded kernels').
template <int NP>
__device__ __forceinline__ void pinf_eval(const Model<NP>& M, const double a[NP], const double r[NP], NewtonState& s,
                                          const double p[NP], double aS[NP], double rS[NP]) {
  if (!pinf_quick<NP>(M, a, r, s, p, aS, rS)) pinf_eval_general<NP>(M, a, r, s, p, aS, rS);
}

// The Newton step f / df of the seeded kernels.
__device__ __forceinline__ double newton_step(const NewtonState& s) {
  double d = qdiv(s.f, s.df, s.ydf);
  if (!(d == d)) d = ndiv(s.f, s.df);
  return d;
}

// RelaxationPInfinite::relaxation src/Relaxations/RelaxationPInfinite.cpp:43-97 with
// RelaxationP::NewtonRaphson src/Relaxations/RelaxationP.cpp:43-68.  a/r/p are the phase state
// after buildPrim (p per phase); the phase sound speeds of that state are needed only by the
// interface-pressure fallback, RelaxationP::computeInterfacePressure :72, recomputed there from
// the same rho_k, p_k as PhaseUEq::extendedCalculusPhase does).  On return a/r hold
// the relaxed state and pstar the relaxed pressure; returns false if the relaxation was skipped.
template <int NP>
__device__ __forceinline__ bool relax_pinf(const Model<NP>& M, double a[NP], double r[NP], const double p[NP],
                                           double& pstar, RelaxStats& st, double seed, bool use_seed,
                                           int max_iter, bool accept = false) {
  st.iters = 0;
  st.fallback = false;
  st.seeded = false;
  st.rejected = false;
  if (M.eps > 1.e-20) {
    bool relax = true;
#pragma unroll
    for (int k = 0; k < NP; k++)
      if (a[k] > (1. - 1.e-5)) relax = false;
    if (!relax) return false;
  }
  double ps = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) ps += a[k] * p[k];
  if (use_seed) {
    // A learned initial guess replaces sum_k alpha_k p_k only when it is finite and inside the
    // bracket of the phase pressures; otherwise it is rejected and the plain start is kept.
    double lo = p[0], hi = p[0];
#pragma unroll
    for (int k = 1; k < NP; k++) { lo = dmin(lo, p[k]); hi = dmax(hi, p[k]); }
    if (isfinite(seed) && seed >= lo && seed <= hi) { ps = seed; st.seeded = true; }
    else st.rejected = true;
  }
  double aS[NP], rS[NP];
  // the first evaluation is at the start itself (f / df = 0 / 1 before it)
  NewtonState s{ps, 0., 1., 1, 1.};
  bool quick = pinf_quick<NP>(M, a, r, s, p, aS, rS);
  while (quick && fabs(s.f) > 1e-10 && s.it < max_iter) {
    const double d = qdiv(s.f, s.df, s.ydf);
    if (!(d == d)) {
      quick = false;
      break;
    }
    s.it++;
    s.ps -= d;
    quick = pinf_quick<NP>(M, a, r, s, p, aS, rS);
  }
  if (!quick) {  // the whole iteration in the general form (the iterates up to here are its own, bit for bit)
    s.ps = ps;
    s.it = 0;
    s.f = 0.;
    s.df = 1.;
    do {
      s.it++;
      s.ps -= ndiv(s.f, s.df);
#pragma unroll
      for (int k = 0; k < NP; k++) s.ps = eos_fix_p(M.eos[k], s.ps);
      pinf_eval_general<NP>(M, a, r, s, p, aS, rS);
    } while (fabs(s.f) > 1e-10 && s.it < max_iter);
  }
  const int iteration = s.it;
  ps = s.ps;
  st.iters = iteration;
  if (iteration < max_iter || accept) {  // accept: a capped iteration keeps its last iterate
#pragma unroll
    for (int k = 0; k < NP; k++) { a[k] = aS[k]; r[k] = rS[k]; }
    pstar = ps;
    return true;
  }
  st.fallback = true;
  double drhodp = 0.;
  double zk[NP], pI = 0., sumZk = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) zk[k] = r[k] * eos_c(M.eos[k], M.eps, r[k], p[k]);
#pragma unroll
  for (int k = 0; k < NP; k++) {
    sumZk += zk[k];
    double sumZj = 0.;
#pragma unroll
    for (int j = 0; j < NP; j++)
      if (j != k) sumZj += zk[j];
    pI += sumZj * (p[k] - 0.);
  }
  pI = ndiv(pI, sumZk * (NP - 1));
#pragma unroll
  for (int k = 0; k < NP; k++) pI = eos_fix_p(M.eos[k], pI);
#pragma unroll
  for (int k = 0; k < NP; k++) {
    double rr = eos_rho_pfinal(M.eos[k], M.eps, p[k], r[k], pI, &drhodp);
    a[k] = ndiv(a[k] * r[k], rr);
    r[k] = rr;
  }
  pstar = pI;
  return true;
}


// ------------------------------------------------------------------ logarithm of the saturation solve
// The saturation temperature solve (Mixture::computeTsat) branches on tight tests (pure-phase
// hypotheses, |f| > 1e-10), so a last-ulp difference between the device's log and the host libm's can
// change a cell's path.  It takes its logarithms from elog (ecg_pow.cuh): ln x carried as a
// double-double from a 128-row table and rounded once, i.e. the correctly rounded logarithm except
// within about 2^-75 of a midpoint; on the solve's arguments (temperatures, pressures) it equals the
// host glibc log on every one of 8e6 tested values.

// ------------------------------------------------------------------ relaxation (p-T-mu, 2 phases)

template <int NP>
__device__ __forceinline__ bool pinf_applies(const Model<NP>& M, const double a[NP]) {
  if (M.eps > 1.e-20) {
#pragma unroll
    for (int k = 0; k < NP; k++)
      if (a[k] > (1. - 1.e-5)) return false;
  }
  return true;
}

// First evaluation at the plain start sum_k alpha_k p_k (relax_pinf's first iteration).
template <int NP>
__device__ __forceinline__ void pinf_first(const Model<NP>& M, const double a[NP], const double r[NP],
                                           const double p[NP], NewtonState& s, double aS[NP], double rS[NP]) {
  double ps = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) ps += a[k] * p[k];
  s.ps = ps;
  s.it = 1;
  pinf_eval<NP>(M, a, r, s, p, aS, rS);
}

// Continues from state s to |f| <= 1e-10 or the cap; relaxes a, r like relax_pinf.
template <int NP>
__device__ __forceinline__ void pinf_finish(const Model<NP>& M, double a[NP], double r[NP], const double p[NP],
                                            NewtonState s, double aS[NP], double rS[NP], double& pstar, RelaxStats& st,
                                            int max_iter, bool accept = false) {
  while (fabs(s.f) > 1e-10 && s.it < max_iter) {
    s.it++;
    s.ps -= newton_step(s);
    pinf_eval<NP>(M, a, r, s, p, aS, rS);
  }
  st.iters = s.it;
  if (s.it < max_iter || accept) {
#pragma unroll
    for (int k = 0; k < NP; k++) { a[k] = aS[k]; r[k] = rS[k]; }
    pstar = s.ps;
    return;
  }
  st.fallback = true;
  double drhodp = 0.;
  double zk[NP], pI = 0., sumZk = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) zk[k] = r[k] * eos_c(M.eos[k], M.eps, r[k], p[k]);
#pragma unroll
  for (int k = 0; k < NP; k++) {
    sumZk += zk[k];
    double sumZj = 0.;
#pragma unroll
    for (int j = 0; j < NP; j++)
      if (j != k) sumZj += zk[j];
    pI += sumZj * (p[k] - 0.);
  }
  pI = ndiv(pI, sumZk * (NP - 1));
#pragma unroll
  for (int k = 0; k < NP; k++) pI = eos_fix_p(M.eos[k], pI);
#pragma unroll
  for (int k = 0; k < NP; k++) {
    double rr = eos_rho_pfinal(M.eos[k], M.eps, p[k], r[k], pI, &drhodp);
    a[k] = ndiv(a[k] * r[k], rr);
    r[k] = rr;
  }
  pstar = pI;
}

// Iteration counts of one p-T-mu relaxation (diagnostics; they do not change the arithmetic).
struct PtmuCount {
  unsigned int solve = 0;      // 1 when the saturation Newton on p* ran
  unsigned int outer = 0;      // its iterations
  unsigned int tsat_calls = 0;  // T_sat(p) solves (pure-phase tests included)
  unsigned int tsat_iters = 0;  // their Newton iterations
  unsigned int tsat_max = 0;    // the largest of them
  unsigned int seeded = 0;      // 1 when the saturation Newton started from a learned (p*, T) seed
  unsigned int rejected = 0;    // 1 when a learned seed was rejected (plain start)
  double pstar = 0., tsat = 0.;  // converged p* and T_sat(p*) of the saturation Newton (recording)
};

// Mixture::computeTsat src/Models/Mixture.cpp:59-100 (liquid and vapour IG/SG).
// T0 > 0: the Newton iteration starts there instead of at 0.1 B / C (a seeded p-T-mu relaxation).
// With B / C > 0, f(T) = A + B / T + C ln T - ... is monotone and of one curvature on (0, B / C), the
// branch the cold start 0.1 B / C converges on: a start left of the root approaches it monotonically, a
// start right of it jumps left of it in one step, possibly past T = 0.  So a start is taken only inside
// (0, 0.5 B / C), and an iterate that leaves (0, B / C) sends the iteration back to the cold start
// (at most once); either way it converges to the root the reference's iteration finds.
__device__ __forceinline__ double compute_tsat(const PtmuParams& t, double p, double* dTsat, bool& err,
                                               PtmuCount* pc = nullptr, double T0 = -1.) {
  const double piL = (t.liq.type == ECG_EOS_IG) ? 0. : t.liq.pinf, piV = (t.vap.type == ECG_EOS_IG) ? 0. : t.vap.pinf;
  int iteration = 0;
  bool seeded = T0 > 0. && T0 < t.half;
  double Tsat = seeded ? T0 : t.cold, f = 0., df = 1., step = 0.;
  // ln(p + pInf) of both phases do not depend on the iterate: evaluated once per solve (the same
  // values enter the same sum, so f has the bits of the reference's per-iteration evaluation)
  const double lnV = elog(p + piV), lnL = t.D * elog(p + piL);
  // the cold start's terms come with the parameters: one iterate less in each solve, of six or seven (measured, p-T-mu
  // expansion 1024^2: cell kernels 0.347 -> 0.341 ms)
  if (!seeded) {
    iteration = 1;
    f = t.f0 - lnV + lnL;
    df = t.df0;
    step = ndiv(f, df);
  }
  if (seeded || fabs(f) > 1e-10) do {
    Tsat -= step;
    if (seeded && !(Tsat > 0. && Tsat < t.branch)) {  // a seeded iterate left the root's branch
      seeded = false;
      Tsat = t.cold;
    }
    iteration++;
    if (iteration > 50) {
      err = true;
      break;
    }
    // B/T, C/T and B/T^2 from one reciprocal (1/T^2 is its square); zero, infinite and NaN iterates make the
    // derivative NaN and take the general quotients
    const double y = nrcp(Tsat), T2 = Tsat * Tsat;
    double bT = qdiv(t.B, Tsat, y);
    df = qdiv(t.C, Tsat, y) - qdiv(t.B, T2, y * y);
    if (!(df == df)) {
      bT = ndiv(t.B, Tsat);
      df = ndiv(t.C, Tsat) - ndiv(t.B, T2);
    }
    f = t.A + bT + t.C * elog(Tsat) - lnV + lnL;
    step = ndiv(f, df);
  } while (fabs(f) > 1e-10);
  if (pc) {
    pc->tsat_calls++;
    pc->tsat_iters += (unsigned int)iteration;
    pc->tsat_max = max(pc->tsat_max, (unsigned int)iteration);
  }
  double dfdp = ndiv(-1., p + piV) + ndiv(t.D, p + piL);
  *dTsat = ndiv(-dfdp, df);
  return Tsat;
}

// computeDensitySaturation (EosIG.cpp:170, EosSG.cpp:172, EosNASG.cpp:189)
__device__ __forceinline__ double eos_rho_sat(const EosParams& q, double eps, double p, double Tsat, double dTsat,
                                              double* drhodp) {
  double pp = (q.type == ECG_EOS_IG) ? p : p + q.pinf;
  double g1cvT = q.gm1 * q.cv * Tsat;
  double den = (q.type == ECG_EOS_NASG) ? g1cvT + q.b * (p + q.pinf) : g1cvT;
  double d = q.gm1 * q.cv * Tsat - pp * q.gm1 * q.cv * dTsat;
  *drhodp = ndiv(d, dmax(den * den, eps));
  return ndiv(pp, dmax(den, eps));
}

// computeDensityEnergySaturation (EosIG.cpp:184, EosSG.cpp:186, EosNASG.cpp:203)
__device__ __forceinline__ double eos_rhoe_sat(const EosParams& q, double p, double rho, double drhodp,
                                               double* drhoedp) {
  if (q.type == ECG_EOS_IG) {
    *drhoedp = q.ig + drhodp * q.eref;
    return cdiv(p, q.gm1, q.ig) + rho * q.eref;
  }
  if (q.type == ECG_EOS_SG) {
    *drhoedp = q.ig + drhodp * q.eref;
    return cdiv(p + q.gpinf, q.gm1, q.ig) + rho * q.eref;
  }
  *drhoedp = cdiv(1. - rho * q.b, q.gm1, q.ig) + drhodp * (q.eref - cdiv(q.b * (p + q.gpinf), q.gm1, q.ig));
  return cdiv((p + q.gpinf) * (1. - rho * q.b), q.gm1, q.ig) + rho * q.eref;
}

// RelaxationPTMu::relaxation src/Relaxations/RelaxationPTMu.cpp:73-200.  rhomix / emix are the
// mixture density and internal energy the cell holds at that point (from buildPrim).  Returns true
// when the phases were updated (the reference then calls fulfillState, so the mixture density
// is recomputed from the new phases).
//
// Seeded forms: T_seed > 0: the T_sat(p) solves of the saturation Newton start at T_seed (the first)
// and then at the previous iteration's T_sat, instead of the cold start 0.1 B / C of every solve (the
// pure-phase tests keep the cold start, so they decide as the reference does); p_seed > 0: the Newton
// iteration on p* starts at p_seed instead of sum_k alpha_k p_k.  Every loop still stops at
// |f| <= 1e-10.
template <int NP>
__device__ __forceinline__ bool relax_ptmu(const Model<NP>& M, const PtmuParams& t, int liq, double pcrit, double a[NP],
                                           double r[NP], double p[NP], double rhomix, double emix, bool& err,
                                           PtmuCount* pc = nullptr, double p_seed = -1., double T_seed = -1.) {
  const EosParams& EL = t.liq;
  const EosParams& EV = t.vap;
  const bool first = liq == 0;  // the liquid is phase 0 (two phases; no run-time index into the phase arrays)
  // (liquid, vapour) values of a phase array
  auto put = [&](double x[NP], double l, double v) {
    x[0] = first ? l : v;
    x[1] = first ? v : l;
  };
  double pStar = 0., Tsat, dTsat = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) pStar += a[k] * p[k];
  if (pStar > pcrit) return false;
  double rho = rhomix, rhoe = rho * emix;
  double pv = eos_p(EV, M.eps, rho, emix);
  double Tv = eos_T(EV, M.eps, rho, pv);
  if (pv > 0) {
    Tsat = compute_tsat(t, pv, &dTsat, err, pc);
    if (Tv >= Tsat) {
      put(a, 0., 1.);
      put(r, first ? r[0] : r[1], rho);
      put(p, first ? p[0] : p[1], pv);
      return true;
    }
  }
  double pl = eos_p(EL, M.eps, rho, emix);
  double Tl = eos_T(EL, M.eps, rho, pl);
  if (pl > 0.) {
    Tsat = compute_tsat(t, pl, &dTsat, err, pc);
    if (Tl <= Tsat) {
      put(a, 1., 0.);
      put(r, rho, first ? r[1] : r[0]);
      put(p, pl, first ? p[1] : p[0]);
      return true;
    }
  }
  double rhoLSat = 0., rhoVSat = 0., drhoLSat, drhoVSat, aLSat = 0., aVSat = 0., daLSat, daVSat;
  double rhoeLSat, rhoeVSat, drhoeLSat, drhoeVSat;
  int iteration = 0;
  double f = 0., df = 1.;
  double Tstart = T_seed;  // start of the next T_sat solve (seeded form)
  if (p_seed > 0.) pStar = p_seed;
  do {
    pStar -= ndiv(f, df);
    iteration++;
    if (iteration > 50) {
      err = true;
      break;
    }
#pragma unroll
    for (int k = 0; k < NP; k++) pStar = eos_fix_p(M.eos[k], pStar);
    Tsat = compute_tsat(t, pStar, &dTsat, err, pc, Tstart);
    if (T_seed > 0.) Tstart = Tsat;
    rhoLSat = eos_rho_sat(EL, M.eps, pStar, Tsat, dTsat, &drhoLSat);
    rhoVSat = eos_rho_sat(EV, M.eps, pStar, Tsat, dTsat, &drhoVSat);
    aLSat = ndiv(rho - rhoVSat, rhoLSat - rhoVSat);
    daLSat = ndiv(-drhoVSat * (rhoLSat - rhoVSat) - (rho - rhoVSat) * (drhoLSat - drhoVSat),
                  (rhoLSat - rhoVSat) * (rhoLSat - rhoVSat));
    aVSat = 1. - aLSat;
    daVSat = -daLSat;
    f = rhoe;
    df = 0.;
    rhoeLSat = eos_rhoe_sat(EL, pStar, rhoLSat, drhoLSat, &drhoeLSat);
    rhoeVSat = eos_rhoe_sat(EV, pStar, rhoVSat, drhoVSat, &drhoeVSat);
    f -= (aLSat * rhoeLSat + aVSat * rhoeVSat);
    df -= (daLSat * rhoeLSat + aLSat * drhoeLSat + daVSat * rhoeVSat + aVSat * drhoeVSat);
    f = ndiv(f, rhoe);
    df = ndiv(df, rhoe);
  } while (fabs(f) > 1e-10);
  if (pc) {
    pc->solve = 1;
    pc->outer = (unsigned int)iteration;
    pc->pstar = pStar;
    pc->tsat = Tsat;
  }
  put(a, aLSat, aVSat);
  put(r, rhoLSat, rhoVSat);
  put(p, pStar, pStar);
  return true;
}

// ------------------------------------------------------------------ energy correction

// Cell::correctionEnergy src/Order1/Cell.cpp:327: MixUEq::totalEnergyToInternalEnergy :175 then
// FluxPUEq::correctionEnergy src/Models/PUEq/FluxPUEq.cpp:68-112 (mixture-EOS pressure).
template <int NP>
__device__ __forceinline__ double correction_pressure(const Model<NP>& M, const double a[NP], const double r[NP],
                                                      double rhomix, double E, double usq) {
  double e = E - 0.5 * usq;
  double rhoe = rhomix * e;
  double pp = rhoe, denom = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const EosParams& q = M.eos[k];
    const double gpi = q.gpi, ig = q.ig;  // sendSpecialMixtureEos constants, computed on the host
    double cov = (q.type == ECG_EOS_NASG) ? q.b : 0.;
    pp -= a[k] * (gpi * (1. - r[k] * cov) + r[k] * q.eref);
    denom += a[k] * ig * (1. - r[k] * cov);
  }
  return ndiv(pp, denom);
}

}  // namespace ecg
