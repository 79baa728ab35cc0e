// Device functions of the temperature-pressure-velocity equilibrium model (PTUEq): a completed face side, HLLC, the
// cell update, and the model in split form (ecg_flow_split.cuh), used by the fused kernels (ecg_step_ptueq.cu) and by
// the split ones (ecg_flow_ptueq_2d.cu, ecg_flow_ptueq_3d.cu).
#pragma once
#include "ecg_flow_split.cuh"

namespace ecg {

struct PtEos {
  EosParams e[2];
};

// Eos::getPInf: the ideal gas has none (Errors::defaultDouble = 0).
__device__ __forceinline__ double pt_pinf(const EosParams& q) { return q.type == ECG_EOS_IG ? 0. : q.pinf; }

// computeDensity(p, T) of an IG or SG phase (EosIG.cpp:85, EosSG.cpp:87).
__device__ __forceinline__ double pt_rho(const EosParams& q, double p, double T) {
  const double den = dmax((q.gm1 * q.cv * T), 0.);
  return q.type == ECG_EOS_IG ? ndiv(p, den) : ndiv(p + q.pinf, den);
}

// One side of a face (or a cell) with its derived quantities.
struct PtSide {
  double a[2], r[2];
  double p, T, rho, e, c;
  double u[3];
};

// ModPTUEq::fulfillState + MixPTUEq::computeMixtureVariables (mass fractions without a floor).
__device__ __forceinline__ void pt_complete(const PtEos& M, PtSide& s) {
  double ek[2], ck[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    s.r[k] = pt_rho(M.e[k], s.p, s.T);
    ek[k] = eos_e(M.e[k], 0., s.r[k], s.p);
    ck[k] = eos_c(M.e[k], 0., s.r[k], s.p);
  }
  s.rho = 0.;
#pragma unroll
  for (int k = 0; k < 2; k++) s.rho += s.a[k] * s.r[k];
  double Y[2];
#pragma unroll
  for (int k = 0; k < 2; k++) Y[k] = ndiv(s.a[k] * s.r[k], s.rho);
  s.e = 0.;
  s.c = 0.;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    s.e += Y[k] * ek[k];
    s.c += Y[k] * ck[k] * ck[k];
  }
  s.c = dsqrt(s.c);
}

// ModPTUEq::solveRiemannIntern src/Models/PTUEq/ModPTUEq.cpp:113-227 on face-frame velocities;
// the total energy uses the face-frame squared norm, as the reference's projected buffer cells do.
__device__ __forceinline__ void hllc_pt(const PtSide& L, const double ul[3], const PtSide& R, const double ur[3],
                                        bool stretched, double dxL, double dxR, double& wmax, double Fm[2], double Fn[3],
                                        double& FE) {
  const double uL = ul[0], cL = L.c, pL = L.p, rhoL = L.rho;
  const double uR = ur[0], cR = R.c, pR = R.p, rhoR = R.rho;
  const double sL = dmin(uL - cL, uR - cR);
  const double sR = dmax(uR + cR, uL + cL);
  wave_add(wmax, stretched, sL, dxL);
  wave_add(wmax, stretched, sR, dxR);
  const double mL = rhoL * (sL - uL), mR = rhoR * (sR - uR);
  double sM = ndiv(pR - pL + mL * uL - mR * uR, mL - mR);
  if (fabs(sM) < 1.e-8) sM = 0.;
  if (sL >= 0.) {
#pragma unroll
    for (int k = 0; k < 2; k++) Fm[k] = L.a[k] * L.r[k] * uL;
    const double Et = L.e + 0.5 * (ul[0] * ul[0] + ul[1] * ul[1] + ul[2] * ul[2]);
    Fn[0] = rhoL * uL * uL + pL;
    Fn[1] = rhoL * ul[1] * uL;
    Fn[2] = rhoL * ul[2] * uL;
    FE = (rhoL * Et + pL) * uL;
  } else if (sR <= 0.) {
#pragma unroll
    for (int k = 0; k < 2; k++) Fm[k] = R.a[k] * R.r[k] * uR;
    const double Et = R.e + 0.5 * (ur[0] * ur[0] + ur[1] * ur[1] + ur[2] * ur[2]);
    Fn[0] = rhoR * uR * uR + pR;
    Fn[1] = rhoR * ur[1] * uR;
    Fn[2] = rhoR * ur[2] * uR;
    FE = (rhoR * Et + pR) * uR;
  } else if (sM >= 0.) {
    const double Et = L.e + 0.5 * (ul[0] * ul[0] + ul[1] * ul[1] + ul[2] * ul[2]);
    const double rhoStar = ndiv(mL, sL - sM);
    const double EStar = Et + (sM - uL) * (sM + ndiv(pL, mL));
    const double pStar = mL * (sM - uL) + pL;
#pragma unroll
    for (int k = 0; k < 2; k++) Fm[k] = ndiv(L.a[k] * L.r[k] * (sL - uL), sL - sM) * sM;
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * ul[1] * sM;
    Fn[2] = rhoStar * ul[2] * sM;
    FE = (rhoStar * EStar + pStar) * sM;
  } else {
    const double Et = R.e + 0.5 * (ur[0] * ur[0] + ur[1] * ur[1] + ur[2] * ur[2]);
    const double rhoStar = ndiv(mR, sR - sM);
    const double EStar = Et + (sM - uR) * (sM + ndiv(pR, mR));
    const double pStar = mR * (sM - uR) + pR;
#pragma unroll
    for (int k = 0; k < 2; k++) Fm[k] = ndiv(R.a[k] * R.r[k] * (sR - uR), sR - sM) * sM;
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * ur[1] * sM;
    Fn[2] = rhoStar * ur[2] * sM;
    FE = (rhoStar * EStar + pStar) * sM;
  }
}

// Resident blocks per SM of the split form's 2D kernels (3D: 8).  Measured on the 2048^2 bubble (us per step; face,
// cell blocks): 8, 8 1229; 9, 9 1197; 9, 10 1190; 10, 10 (48 registers) 1186; 10, 8 1205; 8, 12 1218.
#ifndef ECG_PTUEQ_FACE_MINB
#define ECG_PTUEQ_FACE_MINB 10
#endif
#ifndef ECG_PTUEQ_CELL_MINB
#define ECG_PTUEQ_CELL_MINB 10
#endif

// Update of a cell from its accumulated fluxes and its time-n fields (sn, `stride` apart).
template <int DIM, int PASS>
__device__ __forceinline__ void pt_update(const StepParams& P, const PtEos& M, int64_t nn, int64_t cell,
                                          const double* am, const double* amom, double aE, const double* sn,
                                          int64_t stride) {
  constexpr int FP = 2, FT = 3, FU = 4;
  // ---- FluxPTUEq::buildCons (time-n state), Cell::timeEvolution, FluxPTUEq::buildPrim (:125-160) with
  // MixPTUEq::computePressure (:93-122, Le Martelot's analytic p of two IG/SG phases) and
  // computeTemperature (:126-145)
  const double dt = *P.dt;
  const double scale = (PASS == PASS_PRED) ? 0.5 * dt : dt;
  PtSide n0;
  n0.a[0] = sn[0];
  n0.a[1] = sn[stride];
  n0.p = sn[FP * stride];
  n0.T = sn[FT * stride];
  const double En = sn[(FU + DIM) * stride];
  double rhon = 0.;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    n0.r[k] = pt_rho(M.e[k], n0.p, n0.T);
    rhon += n0.a[k] * n0.r[k];
  }
  double m[2];
#pragma unroll
  for (int k = 0; k < 2; k++) m[k] = am[k] * scale + 1. * (n0.a[k] * n0.r[k]);
  double mom[DIM];
#pragma unroll
  for (int d = 0; d < DIM; d++) mom[d] = amom[d] * scale + 1. * (rhon * sn[(FU + d) * stride]);
  const double rE = aE * scale + 1. * (rhon * En);
  const double rhoMel = 0. + m[0] + m[1];
  double u[3] = {0., 0., 0.};
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    u[d] = ndiv(mom[d], rhoMel);
    if (fabs(u[d]) < 1.e-8) u[d] = 0.;
  }
  const double ie = ndiv(rE, rhoMel) - 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  const EosParams& E1 = M.e[0];
  const EosParams& E2 = M.e[1];
  const double pInf1 = pt_pinf(E1), pInf2 = pt_pinf(E2);
  const double Y1 = ndiv(m[0], rhoMel), Y2 = ndiv(m[1], rhoMel);
  const double q = Y1 * E1.eref + Y2 * E2.eref;
  const double cvMel = Y1 * E1.cv + Y2 * E2.cv;
  const double A1 = ndiv(Y1 * (E1.gamma - 1.) * E1.cv, cvMel) * (rhoMel * (ie - q) - pInf1);
  const double A2 = ndiv(Y2 * (E2.gamma - 1.) * E2.cv, cvMel) * (rhoMel * (ie - q) - pInf2);
  const double p = 0.5 * (A1 + A2 - (pInf1 + pInf2)) +
                   dsqrt(0.25 * (A2 - A1 - (pInf2 - pInf1)) * (A2 - A1 - (pInf2 - pInf1)) + A1 * A2);
  double Tm = 0.;
  Tm += ndiv(ndiv(m[0], rhoMel) * (E1.gamma - 1.) * E1.cv, p + pInf1);
  Tm += ndiv(ndiv(m[1], rhoMel) * (E2.gamma - 1.) * E2.cv, p + pInf2);
  Tm = ndiv(1., Tm * rhoMel);
  P.out[cell] = ndiv(m[0], pt_rho(E1, p, Tm));
  P.out[nn + cell] = ndiv(m[1], pt_rho(E2, p, Tm));
  P.out[(int64_t)FP * nn + cell] = p;
  P.out[(int64_t)FT * nn + cell] = Tm;
#pragma unroll
  for (int d = 0; d < DIM; d++) P.out[(int64_t)(FU + d) * nn + cell] = u[d];
  if (PASS != PASS_PRED) P.out[(int64_t)(FU + DIM) * nn + cell] = ndiv(rE, rhoMel);
}

// The model in split form (ecg_flow_split.cuh).
struct PtFlow {
  using Eos = PtEos;
  struct Side {
    PtSide s;  // s.u unused: the face-frame velocities are ul
    double c, ul[3];
  };
  static constexpr int NM = 2, U = 4, STORED = 0, FACE_MINB = ECG_PTUEQ_FACE_MINB, CELL_MINB = ECG_PTUEQ_CELL_MINB;
  static __device__ __forceinline__ void complete(const Eos& M, Side& A) {
    pt_complete(M, A.s);
    A.c = A.s.c;
  }
  template <int DIM>
  static __device__ __forceinline__ void fields(const double* sq, int RS, int rc, int pn, int p1, int p2, Side& A) {
    A.s.a[0] = sq[rc];
    A.s.a[1] = sq[RS + rc];
    A.s.p = sq[2 * RS + rc];
    A.s.T = sq[3 * RS + rc];
    A.ul[0] = sq[(U + pn) * RS + rc];
    A.ul[1] = sq[(U + p1) * RS + rc];
    A.ul[2] = DIM > 2 ? sq[(U + p2) * RS + rc] : 0.;
  }
  template <int DIM>
  static __device__ __forceinline__ void load(const Eos& M, const double* sq, int RS, int rc, int, int pn, int p1,
                                              int p2, bool, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
    complete(M, A);
  }
  // extrapolation and PhasePTUEq::verifyAndCorrectPhase (alpha in [1e-10, 1 - 1e-10])
  template <int DIM>
  static __device__ __forceinline__ void extrapolate(const Eos& M, const double* sq, int RS, int rc, const double* ssl,
                                                     int SS, int e, int, int pn, int p1, int p2, double dist,
                                                     double sign, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      double a = A.s.a[k] + (sign * ssl[k * SS + e]) * dist;
      if (a < 1e-10) a = 1e-10;
      if (a > 1. - 1e-10) a = 1. - 1e-10;
      A.s.a[k] = a;
    }
    A.s.p += (sign * ssl[2 * SS + e]) * dist;
    A.s.T += (sign * ssl[3 * SS + e]) * dist;
    A.ul[0] += (sign * ssl[(U + pn) * SS + e]) * dist;
    A.ul[1] += (sign * ssl[(U + p1) * SS + e]) * dist;
    if (DIM > 2) A.ul[2] += (sign * ssl[(U + p2) * SS + e]) * dist;
    complete(M, A);
  }
  // symmetry sides are first order only
  template <int DIM, bool O2>
  static __device__ __forceinline__ void wall(const Eos& M, const double* sq, int RS, int rc, const double*, int, int,
                                              int, int pn, int p1, int p2, double, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
    complete(M, A);
  }
  // ModPTUEq::solveRiemannWall src/Models/PTUEq/ModPTUEq.cpp:233-265
  static __device__ __forceinline__ double wall_flux(const Side& A, double sL) {
    return A.s.rho * (A.ul[0] - sL) * A.ul[0] + A.s.p;
  }
  static __device__ __forceinline__ void hllc(const Side& A, const Side& B, bool stretched, double dxL, double dxR,
                                              double& wmax, double Fm[2], double Fn[3], double& FE) {
    hllc_pt(A.s, A.ul, B.s, B.ul, stretched, dxL, dxR, wmax, Fm, Fn, FE);
  }
  template <int DIM, int PASS>
  static __device__ __forceinline__ void update(const StepParams& P, const Eos& M, int64_t nn, int64_t cell,
                                                const double* acc, const double* sn, int64_t stride) {
    pt_update<DIM, PASS>(P, M, nn, cell, acc, acc + 2, acc[2 + DIM], sn, stride);
  }
};

// One pass in split form (the context holds face arrays); a unit per dimension, so that a context loads the code of
// its own kernels only.
template <int DIM>
cudaError_t ptueq_flow(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, cudaStream_t s,
                       bool prepare) {
  PtEos M;
  for (int k = 0; k < 2; k++) M.e[k] = make_eos_params(eos[k]);
  return flow_pass<PtFlow, DIM>(pass, P, G, M, s, prepare);
}
cudaError_t ptueq_flow_2d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, cudaStream_t s,
                          bool prepare);
cudaError_t ptueq_flow_3d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, cudaStream_t s,
                          bool prepare);

}  // namespace ecg
