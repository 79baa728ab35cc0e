// Check of the step kernels' quick forms against their general ones, bit for bit, on hashed states: the Newton
// evaluation of the pressure relaxation (pinf_quick inside relax_pinf against an iteration of
// pinf_eval_general) and the internal face (hllc_quick against fulfill and hllc).  The states span ordinary
// liquids and gases and, mixed in, what sends a cell or a face to the general form: pressures at and below the
// EOS floors, densities at theirs, volume fractions of 0 and 1, tension, zeros, infinities and NaN.  Left out of the
// differences, and counted: the quotients ecg_ieee.cuh excepts, a finite non-zero power of two (alpha_k rho_k) over a
// divisor whose significand is all ones (rho_k*).
#include <cuda_runtime.h>

#include "../csrc/ecg_device.cuh"

using namespace ecg;

namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

struct Draw {
  uint64_t h;
  __device__ double uni() {
    h = mix64(h);
    return (double)(h >> 11) * 0x1p-53;
  }
  __device__ double log10(double lo, double hi) { return exp10(lo + (hi - lo) * uni()); }
};

constexpr long long ALL_ONES = 0xFFFFFFFFFFFFFll;
__device__ __forceinline__ long long significand(double x) { return __double_as_longlong(x) & ALL_ONES; }

// same value, NaN equal to NaN (the sign of a zero may differ)
__device__ __forceinline__ bool same(double x, double y) { return (x != x && y != y) || x == y; }

__device__ double odd_value(Draw& d) {
  const double v[10] = {0., -0., 1e-15, -1e300, 1e300, 1e-300, 1., __longlong_as_double(0x7ff0000000000000ll),
                        __longlong_as_double(0xfff0000000000000ll), __longlong_as_double(0x7ff8000000000000ll)};
  return v[(int)(d.uni() * 10.)];
}

template <int NP>
__device__ void draw_phases(const Model<NP>& M, Draw& d, bool odd, double a[NP], double r[NP], double p[NP]) {
  double s = 0.;
  for (int k = 0; k < NP; k++) {
    const double u = d.uni();
    a[k] = u < 0.3 ? 1e-6 * d.uni() : (u < 0.35 ? 1e-14 : d.uni());
    s += a[k];
  }
  const double p0 = d.uni() < 0.7 ? d.log10(2., 9.5) : -d.log10(2., 8.);
  for (int k = 0; k < NP; k++) {
    a[k] /= s;
    r[k] = M.eos[k].type == ECG_EOS_IG ? d.log10(-4., 2.5) : 900. + 300. * d.uni();
    p[k] = eos_fix_p(M.eos[k], p0 * (d.uni() < 0.5 ? 1. : d.log10(-1., 1.)));
    phase_fix_ar(M.eps, a[k], r[k]);
  }
  if (odd) {
    const int k = (int)(d.uni() * NP), w = (int)(d.uni() * 3.);
    (w == 0 ? a : (w == 1 ? r : p))[k] = odd_value(d);
  }
}

template <int NP>
__global__ void k_quick(uint64_t seed, int iters, Model<NP> M, unsigned long long* out) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long n = 0, bad_newton = 0, bad_face = 0, quick = 0, ties = 0;
  for (int it = 0; it < iters; it++) {
    Draw d{mix64(seed ^ (t * 0x100000001B3ull + (uint64_t)it))};
    const bool odd = d.uni() < 0.1;
    n++;
    {  // pressure relaxation
      double a[NP], r[NP], p[NP], b[NP], q[NP], aS[NP], rS[NP], ps = 0.;
      draw_phases<NP>(M, d, odd, a, r, p);
      for (int k = 0; k < NP; k++) {
        b[k] = a[k];
        q[k] = r[k];
        ps += a[k] * p[k];
      }
      NewtonState s{ps, 0., 1., 0, 1.};
      do {
        s.it++;
        s.ps -= ndiv(s.f, s.df);
        for (int k = 0; k < NP; k++) s.ps = eos_fix_p(M.eos[k], s.ps);
        pinf_eval_general<NP>(M, a, r, s, p, aS, rS);
      } while (fabs(s.f) > 1e-10 && s.it < 100);
      double pstar = 0.;
      RelaxStats st;
      if (relax_pinf<NP>(M, b, q, p, pstar, st, 0., false, 100, true)) {
        bool tie = false, ok = st.iters == s.it && same(pstar, s.ps);
        for (int k = 0; k < NP; k++) {
          const double ar = a[k] * r[k];
          tie = tie || (ar != 0. && isfinite(ar) && significand(ar) == 0 &&
                        (significand(q[k]) == ALL_ONES || significand(rS[k]) == ALL_ONES));
          ok = ok && same(b[k], aS[k]) && same(q[k], rS[k]);
        }
        if (tie) ties++;
        else if (!ok) bad_newton++;
      }
    }
    {  // internal face
      Thermo<NP> L, R, A, B;
      draw_phases<NP>(M, d, odd, L.a, L.r, L.p);
      if (d.uni() < 0.5) {
        R = L;
        for (int k = 0; k < NP; k++) {
          R.r[k] *= 1. + 1e-3 * d.uni();
          R.p[k] = eos_fix_p(M.eos[k], R.p[k] * (1. + 1e-2 * d.uni()));
        }
      } else {
        draw_phases<NP>(M, d, false, R.a, R.r, R.p);
      }
      const double um = d.uni() < 0.3 ? d.log10(-9., 1.) : d.log10(0., 4.);
      double ul[3], ur[3];
      for (int i = 0; i < 3; i++) {
        ul[i] = um * (2. * d.uni() - 1.);
        ur[i] = um * (2. * d.uni() - 1.);
      }
      if (odd && d.uni() < 0.2) ul[0] = odd_value(d);
      A = L;
      B = R;
      Flux<NP> F, G;
      double Fn[3], Gn[3], w = 0., v = 0.;
      if (hllc_quick<NP, true>(M, L, ul, R, ur, false, 1., 1., w, Fn, F)) {
        quick++;
        fulfill<NP>(M, A);
        fulfill<NP>(M, B);
        hllc<NP>(M, A, ul, B, ur, false, 1., 1., v, Gn, G);
        bool ok = same(w, v) && same(F.E, G.E) && same(F.sM, G.sM) && same(F.uStar, G.uStar);
        for (int i = 0; i < 3; i++) ok = ok && same(Fn[i], Gn[i]);
        for (int k = 0; k < NP; k++) ok = ok && same(F.a[k], G.a[k]) && same(F.m[k], G.m[k]) && same(F.en[k], G.en[k]);
        if (!ok) bad_face++;
      }
    }
  }
  atomicAdd(out, n);
  atomicAdd(out + 1, bad_newton);
  atomicAdd(out + 2, bad_face);
  atomicAdd(out + 3, quick);
  atomicAdd(out + 4, ties);
}

template <int NP>
cudaError_t run(uint64_t seed, int blocks, int iters, const ecg_eos* eos, double eps, unsigned long long* d) {
  Model<NP> M;
  for (int k = 0; k < NP; k++) M.eos[k] = make_eos_params(eos[k]);
  M.eps = eps;
  k_quick<NP><<<blocks, 128>>>(seed, iters, M, d);
  return cudaGetLastError();
}

}  // namespace

// blocks x 128 threads x iters states of np (2 or 3) phases with the given EOS; counts[0] = states, [1] =
// relaxations and [2] = faces whose results differ, [3] = faces hllc_quick solved, [4] = relaxations left out.
// Returns 0, a CUDA error code, or -1 for arguments outside the limits.
extern "C" int ecg_probe_quick_counts(unsigned long long seed, int np, const ecg_eos* eos, double eps, int blocks, int iters,
                                      unsigned long long counts[5]) {
  if ((np != 2 && np != 3) || !eos || blocks <= 0 || iters <= 0) return -1;
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 5 * sizeof(unsigned long long));
  if (e != cudaSuccess) return (int)e;
  e = cudaMemset(d, 0, 5 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = np == 2 ? run<2>(seed, blocks, iters, eos, eps, d) : run<3>(seed, blocks, iters, eos, eps, d);
  if (e == cudaSuccess) e = cudaMemcpy(counts, d, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}

// The first four of these.
extern "C" int ecg_probe_quick_check(unsigned long long seed, int np, const ecg_eos* eos, double eps, int blocks, int iters,
                                     unsigned long long counts[4]) {
  unsigned long long c[5] = {0, 0, 0, 0, 0};
  const int rc = ecg_probe_quick_counts(seed, np, eos, eps, blocks, iters, c);
  for (int i = 0; i < 4; i++) counts[i] = c[i];
  return rc;
}
