// Device functions of the Euler (single-phase) model: a completed face side, HLLC, the cell update, and the model in
// split form (ecg_flow_split.cuh), used by the fused kernels (ecg_step_euler.cu) and by the split ones
// (ecg_flow_euler_2d.cu, ecg_flow_euler_3d.cu).
#pragma once
#include "ecg_flow_split.cuh"

namespace ecg {

struct EulerSide {
  double rho, p, c, E;
  double u[3];  // absolute frame
};

__device__ __forceinline__ void euler_complete(const EosParams& q, double eps, EulerSide& s) {
  // PhaseEuler::extendedCalculusPhase: e, c, E = e + |u|^2 / 2 (absolute frame)
  double e = eos_e(q, eps, s.rho, s.p);
  s.c = eos_c(q, eps, s.rho, s.p);
  s.E = e + 0.5 * (s.u[0] * s.u[0] + s.u[1] * s.u[1] + s.u[2] * s.u[2]);
}

// Resident blocks per SM of the split form's 2D kernels (3D: 8).  Measured on the 2048^2 blast (us per step; face,
// cell blocks): 8, 8 801; 9, 10 766; 10, 12 744; 12, 8 732; 12, 10 (40 and 48 registers) 720; 14, 12 721.
#ifndef ECG_EULER_FACE_MINB
#define ECG_EULER_FACE_MINB 12
#endif
#ifndef ECG_EULER_CELL_MINB
#define ECG_EULER_CELL_MINB 10
#endif

// ModEuler::solveRiemannIntern src/Models/Euler/ModEuler.cpp:105-225 (strict sL > 0 / sR < 0).
__device__ __forceinline__ void hllc_euler(const EulerSide& L, const double ul[3], const EulerSide& R,
                                           const double ur[3], bool stretched, double dxL, double dxR, double& wmax, double& Fm,
                                           double Fn[3], double& FE, double* sM_out = nullptr) {
  double uL = ul[0], vL = ul[1], wL = ul[2], pL = L.p, rhoL = L.rho, cL = L.c, EL = L.E;
  double uR = ur[0], vR = ur[1], wR = ur[2], pR = R.p, rhoR = R.rho, cR = R.c, ER = R.E;
  double sL = dmin(uL - cL, uR - cR);
  double sR = dmax(uR + cR, uL + cL);
  wave_add(wmax, stretched, sL, dxL);
  wave_add(wmax, stretched, sR, dxR);
  double mL = rhoL * (sL - uL), mR = rhoR * (sR - uR);
  double sM = ndiv(pR - pL + mL * uL - mR * uR, mL - mR);
  if (fabs(sM) < 1.e-8) sM = 0.;
  if (sM_out) *sM_out = sM;
  if (sL > 0.) {
    Fm = rhoL * uL;
    Fn[0] = rhoL * uL * uL + pL;
    Fn[1] = rhoL * vL * uL;
    Fn[2] = rhoL * wL * uL;
    FE = (rhoL * EL + pL) * uL;
  } else if (sR < 0.) {
    Fm = rhoR * uR;
    Fn[0] = rhoR * uR * uR + pR;
    Fn[1] = rhoR * vR * uR;
    Fn[2] = rhoR * wR * uR;
    FE = (rhoR * ER + pR) * uR;
  } else if (sM >= 0.) {
    double pStar = mL * (sM - uL) + pL;
    double rhoStar = ndiv(mL, sL - sM);
    double Estar = EL + (sM - uL) * (sM + ndiv(pL, mL));
    Fm = rhoStar * sM;
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * sM * vL;
    Fn[2] = rhoStar * sM * wL;
    FE = (rhoStar * Estar + pStar) * sM;
  } else {
    double pStar = mR * (sM - uR) + pR;
    double rhoStar = ndiv(mR, sR - sM);
    double Estar = ER + (sM - uR) * (sM + ndiv(pR, mR));
    Fm = rhoStar * sM;
    Fn[0] = rhoStar * sM * sM + pStar;
    Fn[1] = rhoStar * sM * vR;
    Fn[2] = rhoStar * sM * wR;
    FE = (rhoStar * Estar + pStar) * sM;
  }
}

// FluxEuler::buildCons, Cell::timeEvolution, FluxEuler::buildPrim of a cell from its accumulated fluxes and its
// time-n fields (sn, `stride` apart).
template <int DIM, int PASS>
__device__ __forceinline__ void euler_update(const StepParams& P, const EosParams& q, double eps, int64_t nn,
                                             int64_t cell, double am, const double* amom, double aE, const double* sn,
                                             int64_t stride) {
  const double dt = *P.dt;
  const double scale = (PASS == PASS_PRED) ? 0.5 * dt : dt;
  const double rn = sn[0];
  const double En = sn[(2 + DIM) * stride];
  am = am * scale + 1. * rn;
  double u[DIM], usq = 0.;
#pragma unroll
  for (int d = 0; d < DIM; d++) u[d] = amom[d] * scale + 1. * (rn * sn[(2 + d) * stride]);
  aE = aE * scale + 1. * (rn * En);
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    u[d] = ndiv(u[d], am);
    if (fabs(u[d]) < 1.e-8) u[d] = 0.;
    usq += u[d] * u[d];
  }
  const double E = ndiv(aE, am);
  const double p = eos_p(q, eps, am, E - 0.5 * usq);
  P.out[cell] = am;
  P.out[nn + cell] = p;
#pragma unroll
  for (int d = 0; d < DIM; d++) P.out[(int64_t)(2 + d) * nn + cell] = u[d];
  if (PASS != PASS_PRED) P.out[(int64_t)(2 + DIM) * nn + cell] = E;
}

// The model in split form (ecg_flow_split.cuh); the energy of a completed side sums |u|^2 in the absolute
// frame's order.
struct EulerFlow {
  struct Eos {
    EosParams q;
    double eps;
  };
  struct Side {
    EulerSide s;  // s.u unused: the face-frame velocities are ul
    double c, ul[3];
  };
  static constexpr int NM = 1, U = 2, STORED = 1, FACE_MINB = ECG_EULER_FACE_MINB, CELL_MINB = ECG_EULER_CELL_MINB;
  static __device__ __forceinline__ void complete(const Eos& M, int ax, Side& A) {
    const double n2 = A.ul[0] * A.ul[0], t1 = A.ul[1] * A.ul[1], t2 = A.ul[2] * A.ul[2];
    const double e = eos_e(M.q, M.eps, A.s.rho, A.s.p);
    A.c = A.s.c = eos_c(M.q, M.eps, A.s.rho, A.s.p);
    A.s.E = e + 0.5 * (ax == 2 ? (t1 + t2) + n2 : (n2 + t1) + t2);
  }
  template <int DIM>
  static __device__ __forceinline__ void fields(const double* sq, int RS, int rc, int pn, int p1, int p2, Side& A) {
    A.s.rho = sq[rc];
    A.s.p = sq[RS + rc];
    A.ul[0] = sq[(U + pn) * RS + rc];
    A.ul[1] = sq[(U + p1) * RS + rc];
    A.ul[2] = DIM > 2 ? sq[(U + p2) * RS + rc] : 0.;
  }
  template <int DIM>
  static __device__ __forceinline__ void load(const Eos& M, const double* sq, int RS, int rc, int ax, int pn, int p1,
                                              int p2, bool stored, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
    complete(M, ax, A);
    if (stored) A.s.E = sq[(U + DIM) * RS + rc];  // no fulfillState on interior first-order faces
  }
  // global limiter (the interface detector never fires for Euler), extrapolation
  template <int DIM>
  static __device__ __forceinline__ void shift(const double* ssl, int SS, int e, int pn, int p1, int p2, double dist,
                                               double sign, Side& A) {
    A.s.rho += (sign * ssl[e]) * dist;
    A.s.p += (sign * ssl[SS + e]) * dist;
    A.ul[0] += (sign * ssl[(U + pn) * SS + e]) * dist;
    A.ul[1] += (sign * ssl[(U + p1) * SS + e]) * dist;
    if (DIM > 2) A.ul[2] += (sign * ssl[(U + p2) * SS + e]) * dist;
  }
  template <int DIM>
  static __device__ __forceinline__ void extrapolate(const Eos& M, const double* sq, int RS, int rc, const double* ssl,
                                                     int SS, int e, int ax, int pn, int p1, int p2, double dist,
                                                     double sign, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
    shift<DIM>(ssl, SS, e, pn, p1, p2, dist, sign, A);
    if (A.s.rho < 1.e-10) A.s.rho = 1.e-10;
    A.s.p = eos_fix_p(M.q, A.s.p);
    eos_rho_max(M.q, A.s.rho);
    complete(M, ax, A);
  }
  // BoundCondWallO2Cartesian::solveRiemann :111-141: extrapolation by the signed distance without clamps
  template <int DIM, bool O2>
  static __device__ __forceinline__ void wall(const Eos& M, const double* sq, int RS, int rc, const double* ssl, int SS,
                                              int e, int ax, int pn, int p1, int p2, double dist, Side& A) {
    fields<DIM>(sq, RS, rc, pn, p1, p2, A);
    if (O2) shift<DIM>(ssl, SS, e, pn, p1, p2, dist, 1., A);
    complete(M, ax, A);
  }
  // ModEuler::solveRiemannWall src/Models/Euler/ModEuler.cpp:368-409
  static __device__ __forceinline__ double wall_flux(const Side& A, double sL) {
    return A.s.rho * A.ul[0] * (A.ul[0] - sL) + A.s.p;
  }
  static __device__ __forceinline__ void hllc(const Side& A, const Side& B, bool stretched, double dxL, double dxR,
                                              double& wmax, double Fm[1], double Fn[3], double& FE) {
    hllc_euler(A.s, A.ul, B.s, B.ul, stretched, dxL, dxR, wmax, Fm[0], Fn, FE);
  }
  template <int DIM, int PASS>
  static __device__ __forceinline__ void update(const StepParams& P, const Eos& M, int64_t nn, int64_t cell,
                                                const double* acc, const double* sn, int64_t stride) {
    euler_update<DIM, PASS>(P, M.q, M.eps, nn, cell, acc[0], acc + 1, acc[1 + DIM], sn, stride);
  }
};

// One pass in split form (the context holds face arrays); a unit per dimension, so that a context loads the code of
// its own kernels only.
template <int DIM>
cudaError_t euler_flow(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, double eps, cudaStream_t s,
                       bool prepare) {
  return flow_pass<EulerFlow, DIM>(pass, P, G, EulerFlow::Eos{make_eos_params(eos[0]), eps}, s, prepare);
}
cudaError_t euler_flow_2d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, double eps,
                          cudaStream_t s, bool prepare);
cudaError_t euler_flow_3d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, double eps,
                          cudaStream_t s, bool prepare);

}  // namespace ecg
