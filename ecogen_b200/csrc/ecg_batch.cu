// Batched independent 1D cases: every pass is one face-flux kernel and one cell kernel over all cases.
//
// The reference runs independent cases one after the other (src/main.cpp:82-133), each with its
// own time loop.  Here all cases live in one concatenated structure-of-arrays state (case c owns
// cells [off_c, off_c + n_c)), every pass (first order, or MUSCL predictor then corrector) is two launches
// over lists of (case, first face) and (case, first cell) items, one block per item (where the face fluxes do
// not all fit the free memory: two launches per piece of the batch), and each case keeps its own dt: the fastest wave of an item's faces merges into the
// case's slot with one atomicMin (a segmented min-reduction), then a per-case update sets
// dt_c = cfl_c dtMax_c.  The step sequence is captured once as a CUDA graph.  The faces of an item (the
// tile) are picked by a small autotuner that times each candidate on a copy of the state.
//
// Why two kernels: one kernel per pass (persistent blocks over a queue of tiles) held the face work, the
// cell update and the seeded update at once, spilled 1.1 KB a thread at 80 registers and met four barriers
// per tile, at which warps waited for the slowest cell's Newton iteration.  The face fluxes cost
// 160 bytes of HBM traffic per cell and pass, which the passes have to spare.  Measured on one B200
// (4096 two-phase tubes, 8.6 M cells, MUSCL + van Leer, mid-run states, host copies of a 40-step pass
// included): 3.54 -> 3.30 ms per step; 64 tubes (0.13 M cells) 131 -> 111 us.  Same bits.
// Launched as dependents of one another, with the place of an item in the item, u and E copied ahead and the host's
// zero fill of the unused velocities beside the download: 3.06 -> 2.83 ms, 95.6 -> 91.9 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "ecg_internal.h"
#include "ecg_kapila_split.cuh"

// Resident threads per SM asked of the face kernel, in whole blocks: 896 are 14 blocks of 64 or 7 of 128 threads (72
// registers) and 3 of 256 (768 threads, 80 registers, the tile the autotuner picks on large batches).
#ifndef ECG_BATCH_SM_THREADS
#define ECG_BATCH_SM_THREADS 896
#endif

namespace ecg {

struct BatchCase {
  int64_t off;
  int n;
  double dx, coefA, lcfl, cfl;
};

struct BatchScalars {
  double dt, t;
  unsigned long long dtmax_bits;
  long long it;
};

// A block's piece of a case: the faces or cells of case c from `first` on, up to face `end` or cell `end` - 1.  The
// case's size and place stand here too, so that the block's loads start one access earlier than through BatchCase;
// face f's fluxes are at fbase + f.
struct __align__(16) BatchItem {
  int c, first, n, end;
  int64_t off, fbase;
};

struct BatchParams {
  StepParams P;              // q / sn / out point at the concatenated state (stride = total cells)
  const BatchCase* cases;
  BatchScalars* scal;
  const BatchItem* items;    // face items of the face kernel, cell items of the cell kernel
  double* flux;              // face fluxes of a piece of the batch, stride nfaces
  int64_t nfaces;
};

// A face item: TB - 1 faces of one case for TB threads, so that the TB cells whose limited slopes they read
// take one round of the block.
template <int NP, int TB, int PASS, int TYPES>
struct BatchTile {
  static constexpr bool O2 = (PASS != PASS_O1);
  static constexpr bool LSL = O2 && code_limiter(TYPES) >= 0;
  static constexpr int TF = TB - 1;
  static constexpr int H = O2 ? 2 : 1;               // cells staged before the first face
  static constexpr int RL = TF + (O2 ? 3 : 1);
  static constexpr int NA0 = (PASS == PASS_CORR && !LSL) ? 1 : 0;
  static constexpr int SS = O2 ? (LSL ? TF + 1 : TF + 2) : 1;
  static constexpr size_t smem_bytes() {
    return sizeof(double) * ((size_t)RL * (Fields<NP, 1>::NQ + NA0) + (O2 ? (size_t)SS * Fields<NP, 1>::NSL : 0));
  }
};

// Centre of cell g, with the reference's arithmetic.
__device__ __forceinline__ double batch_centre(const BatchCase& C, int g) { return (g + 0.5) * C.dx; }

template <int NP>
__device__ __forceinline__ void store_batch_face(const BatchParams& B, int64_t fid, double mom, const Flux<NP>& F) {
  double* out = B.flux + fid;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    out[(int64_t)k * B.nfaces] = F.a[k];
    out[(int64_t)(NP + k) * B.nfaces] = F.m[k];
    out[(int64_t)(2 * NP + k) * B.nfaces] = F.en[k];
  }
  out[(int64_t)(3 * NP) * B.nfaces] = mom;
  out[(int64_t)(3 * NP + 1) * B.nfaces] = F.E;
  out[(int64_t)(3 * NP + 2) * B.nfaces] = F.sM;
  out[(int64_t)(3 * NP + 3) * B.nfaces] = F.uStar;
}

// The two sides of internal face f, face i of the item; FULFILL: their closure too.
template <int NP, int TB, int PASS, int TYPES, bool FULFILL>
__device__ __forceinline__ void batch_sides(const StepParams& P, const Model<NP>& M, const double* sq, const BatchCase& C,
                                            int n, int f, int i, bool pone, Thermo<NP>& tl, double ul[3], Thermo<NP>& tr,
                                            double ur[3]) {
  using FL = Fields<NP, 1>;
  using K = BatchTile<NP, TB, PASS, TYPES>;
  constexpr int RS = K::RL, SS = K::SS;
  const double* a0 = K::NA0 ? sq + (size_t)FL::NQ * RS : sq;
  const double* ssl = sq + (size_t)(FL::NQ + K::NA0) * RS;
  const int gl = f - 1, rl = i + K::H - 1, rr = rl + 1;
  const double pl = batch_centre(C, gl), pf = pl + 0.5 * C.dx, pr = batch_centre(C, gl + 1);
  if (!K::O2) {
    cell_thermo<NP, 1, FULFILL>(M, sq, RS, rl, tl, ul);
    cell_thermo<NP, 1, FULFILL>(M, sq, RS, rr, tr, ur);
  } else if (K::LSL) {
    extrapolate_side<NP, 1, FULFILL>(M, sq, RS, rl, ssl, SS, i, 0, 0, 0, fabs(pf - pl), 1., pone, tl, ul);
    extrapolate_side<NP, 1, FULFILL>(M, sq, RS, rr, ssl, SS, i + 1, 0, 0, 0, fabs(pf - pr), -1., pone, tr, ur);
  } else {
    const int f1 = i + 1;
    const bool hasL = (gl - 1 >= 0), hasR = (gl + 2 < n);
    const double aL = sq[FL::A * RS + rl], aR = sq[FL::A * RS + rr];
    const double aLL = hasL ? a0[rl - 1] : 0., aRR = hasR ? a0[rr + 1] : 0.;
    constexpr bool kThinc = (TYPES == EOS_DYNAMIC);
    constexpr int kLim = code_limiter(TYPES);
    reconstruct_side<NP, 1, kThinc, kLim, FULFILL>(M, P, sq, RS, rl, ssl, SS, f1, hasL ? i : -1, aL, aR, aLL,
                                                   fabs(pf - pl), 1., tl, ul);
    reconstruct_side<NP, 1, kThinc, kLim, FULFILL>(M, P, sq, RS, rr, ssl, SS, f1, hasR ? i + 2 : -1, aR, aL, aRR,
                                                   fabs(pf - pr), -1., tr, ur);
  }
}

// Any face of an item, sides of the case included, solved by fulfill and hllc and stored; returns its wave value.
template <int NP, int TB, int PASS, int TYPES>
static __device__ __noinline__ double batch_face_general(const BatchParams& B, const Model<NP>& M0, const double* sq,
                                                         const BatchCase C, int64_t fid, int f, int i, bool pone) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);
  using K = BatchTile<NP, TB, PASS, TYPES>;
  double wmax = wave_none(false), Fn[3];
  Flux<NP> F;
  if (f == 0 || f == C.n) {
    // non-reflecting side: HLLC(cell, cell) in the side's frame (BoundCondNonReflecting::
    // solveRiemannBoundary src/BoundConds/BoundCondNonReflecting.cpp:62)
    const bool neg = f == 0;
    Thermo<NP> t;
    double ug[3], ul[3], mom[3];
    cell_thermo<NP, 1>(M, sq, K::RL, neg ? i + K::H : i + K::H - 1, t, ug);
    to_local(0, neg, ug, ul);
    hllc<NP>(M, t, ul, t, ul, false, C.lcfl, C.lcfl, wmax, Fn, F);
    to_global(0, neg, Fn, mom);
    Fn[0] = mom[0];
  } else {
    Thermo<NP> tl, tr;
    double ul[3], ur[3];
    batch_sides<NP, TB, PASS, TYPES, true>(B.P, M, sq, C, C.n, f, i, pone, tl, ul, tr, ur);
    hllc<NP, K::O2>(M, tl, ul, tr, ur, false, C.lcfl, C.lcfl, wmax, Fn, F);
  }
  store_batch_face<NP>(B, fid, Fn[0], F);
  return wmax;
}

template <int NP, int TB, int PASS, int TYPES>
__global__ void __launch_bounds__(TB, ECG_BATCH_SM_THREADS / TB) k_batch_faces(const __grid_constant__ BatchParams B,
                                                                                  const __grid_constant__ Model<NP> M0) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);  // EOS types compiled in for the shipped workload
  using FL = Fields<NP, 1>;
  using K = BatchTile<NP, TB, PASS, TYPES>;
  constexpr bool O2 = K::O2, LSL = K::LSL;
  constexpr int TF = K::TF, RS = K::RL, SS = K::SS;
  extern __shared__ double smem[];
  double* sq = smem;
  double* sa0 = sq + (size_t)FL::NQ * RS;
  double* ssl = sa0 + (size_t)K::NA0 * RS;
  const StepParams& P = B.P;
  const int64_t nn = P.n;
  const int tid = threadIdx.x;
  chain_wait();
  chain_next();
  const BatchItem I = B.items[blockIdx.x];
  const BatchCase& C = B.cases[I.c];
  const int c = I.c, f0 = I.first, n = I.n;
  // ---- stage the cells the item's faces read, f0 - H and up
  for (int e = tid; e < RS; e += TB) {
    const int g = f0 - K::H + e;
    if (g >= 0 && g < n) {
      const int64_t gi = I.off + g;
#pragma unroll
      for (int f = 0; f < FL::NQ; f++) sq[f * RS + e] = P.q[(int64_t)f * nn + gi];
      if (K::NA0) sa0[e] = P.sn[(int64_t)FL::A * nn + gi];
    }
  }
  __syncthreads();
  // centre-to-centre distance of cells g, g + 1 with the reference's arithmetic (Element::distance: sqrt(x x),
  // which is |x| bit for bit)
  auto dist = [&](int g) { return fabs(batch_centre(C, g) - batch_centre(C, g + 1)); };
  bool pone = true;
  if (LSL) {
    double pf = M.eos[0].pfloor;
#pragma unroll
    for (int k = 1; k < NP; k++) pf = dmax(pf, M.eos[k].pfloor);
    for (int e = tid; e < SS; e += TB) {  // limited slopes of cell f0 - 1 + e
      const int g = f0 - 1 + e;
      if (g < 0 || g >= n) continue;
      const int rc = e + 1;
      if (g == 0 || g == n - 1) {  // no face beyond: every limited slope is zero
#pragma unroll
        for (int f = 0; f < FL::NSL; f++) ssl[f * SS + e] = 0.;
        pone = pone && sq[FL::P * RS + rc] >= pf;
        continue;
      }
      const bool one = sq[FL::P * RS + rc - 1] >= pf && sq[FL::P * RS + rc] >= pf && sq[FL::P * RS + rc + 1] >= pf;
      pone = pone && one;
      const double dm = dist(g - 1), dp = dist(g);
      cell_slopes<NP, 1, code_limiter(TYPES)>(M, sq, RS, rc - 1, rc, rc + 1, dm, nrcp(dm), dp, nrcp(dp), one, ssl, SS, e);
    }
    pone = __syncthreads_and(pone);
  } else if (O2) {
    for (int e = tid; e < SS; e += TB) {  // slope e at face f0 - 1 + e
      const int gl = f0 - 2 + e;
      if (gl < 0 || gl + 1 >= n) continue;
      const int rl = e, rr = e + 1;
      const double d = dist(gl);
#pragma unroll
      for (int k = 0; k < NP; k++) {
        ssl[k * SS + e] = ndiv(sq[(FL::A + k) * RS + rr] - sq[(FL::A + k) * RS + rl], d);
        ssl[(NP + k) * SS + e] = ndiv(sq[(FL::R + k) * RS + rr] - sq[(FL::R + k) * RS + rl], d);
        double pR = eos_fix_p(M.eos[k], sq[FL::P * RS + rr]), pL = eos_fix_p(M.eos[k], sq[FL::P * RS + rl]);
        ssl[(2 * NP + k) * SS + e] = ndiv(pR - pL, d);
      }
      ssl[(3 * NP) * SS + e] = ndiv(sq[FL::U * RS + rr] - sq[FL::U * RS + rl], d);
    }
    __syncthreads();
  }
  double wmax = wave_none(false);
  const int f = f0 + tid;
  if (tid < TF && f <= I.end) {
    Thermo<NP> tl, tr;
    double ul[3], ur[3], Fn[3];
    Flux<NP> F;
    bool ok = true;
    if (f > 0 && f < n) {
      batch_sides<NP, TB, PASS, TYPES, false>(P, M, sq, C, n, f, tid, pone, tl, ul, tr, ur);
    } else {  // a non-reflecting side: HLLC(cell, cell) in the side's frame, with the other faces of the warp
      cell_thermo<NP, 1, false>(M, sq, RS, f == 0 ? tid + K::H : tid + K::H - 1, tl, ul);
      if (f == 0) ul[0] = -ul[0];
      tr = tl;
#pragma unroll
      for (int i = 0; i < 3; i++) ur[i] = ul[i];
#pragma unroll
      for (int k = 0; k < NP; k++) ok = ok && tl.r[k] >= 1.e-15;
    }
    const bool solved = hllc_quick<NP, !O2>(M, tl, ul, tr, ur, false, C.lcfl, C.lcfl, wmax, Fn, F, ok);
    if (f == 0) Fn[0] = -Fn[0];
    if (solved) store_batch_face<NP>(B, I.fbase + f, Fn[0], F);
    // operands out of hllc_quick's range
    if (!solved) wmax = dmax(wmax, batch_face_general<NP, TB, PASS, TYPES>(B, M0, sq, C, I.fbase + f, f, tid, pone));
  }
  // ---- segmented reduction: this item's faces belong to case c only
  __shared__ double red[TB / 32];
  double v = wmax;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < TB / 32; w++) v = dmax(v, red[w]);
    atomic_min_pos_double(&B.scal[c].dtmax_bits, wave_dtmax(v, false, C.lcfl));
  }
}

// One thread per cell of an item: the fluxes of its two faces, left added, right subtracted, sides of the case
// last, then the cell update.
template <int NP, int PASS, bool SEED, int TYPES>
__global__ void __launch_bounds__(CELL_THREADS, SEED ? ECG_CELL_SEED_MINB : ECG_CELL_MINB)
    k_batch_cells(BatchParams B, Model<NP> M0) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);
  using FL = Fields<NP, 1>;
  const StepParams& P = B.P;
  const int64_t nn = P.n;
  chain_wait();
  chain_next();
  const BatchItem I = B.items[blockIdx.x];
  const BatchCase& C = B.cases[I.c];
  const int c = I.c, g = I.first + (int)threadIdx.x;
  const bool own = g < I.end;
  const int64_t cell = I.off + g;
  __shared__ double ue[2][CELL_THREADS];  // the time-n u and E, copied ahead
  CellCounters cc;
  CellPrim<NP, 1> cp;
  if (own) {
    double an[NP], rn[NP], pn[NP], aa[NP], am[NP], ae[NP], amom[1] = {0.}, aE = 0.;
    cell_copy(&ue[0][threadIdx.x], P.sn + (int64_t)FL::U * nn + cell);
    cell_copy(&ue[1][threadIdx.x], P.sn + (int64_t)FL::E * nn + cell);
    const double p0 = P.sn[(int64_t)FL::P * nn + cell];
#pragma unroll
    for (int k = 0; k < NP; k++) {
      an[k] = P.sn[(int64_t)(FL::A + k) * nn + cell];
      rn[k] = P.sn[(int64_t)(FL::R + k) * nn + cell];
      pn[k] = eos_fix_p(M.eos[k], p0);
      aa[k] = am[k] = ae[k] = 0.;
    }
    const int64_t fid = I.fbase + g;
    Flux<NP> FA, FB;  // the cell's lower and upper face
    load_face_flux<NP, 1>(B.flux, B.nfaces, fid, FA, P.stats);
    load_face_flux<NP, 1>(B.flux, B.nfaces, fid + 1, FB, P.stats);
    if (g > 0) acc_face<NP, 1>(C.coefA, true, FA, an, pn, aa, am, ae, amom, aE);
    if (g < I.n - 1) acc_face<NP, 1>(C.coefA, false, FB, an, pn, aa, am, ae, amom, aE);
    if (g == 0) acc_face<NP, 1>(C.coefA, false, FA, an, pn, aa, am, ae, amom, aE);
    if (g == I.n - 1) acc_face<NP, 1>(C.coefA, false, FB, an, pn, aa, am, ae, amom, aE);
    cell_copies_wait();
    kapila_rebuild<NP, 1, PASS>(P, M, nn, cell, B.scal[c].dt, an, rn, pn, aa, am, ae, amom, aE, cp,
                                &ue[0][threadIdx.x], CELL_THREADS);
  }
  SeedGate<NP> sg;
  if (SEED) seed_gate<NP, 1>(P, M, own, cp, sg);
  if (own) kapila_finish<NP, 1, PASS, false, SEED, (TYPES == EOS_DYNAMIC)>(P, M, nn, cell, cp, sg, cc);
  // the per-bin histogram is not kept in batched mode (relax_calls / newton_evals / newton_max are)
  block_counters<CELL_THREADS>(P.stats, cc.relax, cc.iters, cc.fallback, cc.seeded, cc.rejected, cc.nonfinite, 0u, cc.iters, false);
}

__global__ void k_batch_finalize(BatchScalars* s, const BatchCase* cases, int ncases) {
  chain_wait();
  chain_next();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncases) return;
  double dtmax = __longlong_as_double((long long)s[c].dtmax_bits);
  s[c].t += s[c].dt;
  s[c].it += 1;
  s[c].dt = cases[c].cfl * dtmax;
  s[c].dtmax_bits = (unsigned long long)__double_as_longlong(1.e10);
}

// One pass: the face kernel over fitems, the cell kernel over citems; with prepare, the face kernel's shared
// memory is configured.
template <int NP, int TB, int PASS, int TYPES>
static cudaError_t batch_one(BatchParams B, const ecg_eos* eos, double eps, const BatchItem* citems, int nf, int nc,
                             cudaStream_t s, bool prepare) {
  auto kern = k_batch_faces<NP, TB, PASS, TYPES>;
  const size_t sm = BatchTile<NP, TB, PASS, TYPES>::smem_bytes();
  if (prepare) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  Model<NP> M;
  for (int k = 0; k < NP; k++) M.eos[k] = make_eos_params(eos[k]);
  M.eps = eps;
  cudaError_t e = launch_chained(kern, dim3(nf), dim3(TB), sm, s, true, B, M);
  if (e != cudaSuccess) return e;
  B.items = citems;
  return launch_chained(B.P.mlp != nullptr ? k_batch_cells<NP, PASS, true, TYPES> : k_batch_cells<NP, PASS, false, TYPES>,
                        dim3(nc), dim3(CELL_THREADS), 0, s, true, B, M);
}

template <int NP, int TB, int TYPES = EOS_DYNAMIC>
static cudaError_t batch_tb(int pass, const BatchParams& B, const ecg_eos* eos, double eps, const BatchItem* citems, int nf,
                            int nc, cudaStream_t s, bool prepare) {
  if constexpr (TYPES == EOS_DYNAMIC)  // the compiled-in configuration is a MUSCL one
    if (pass == PASS_O1) return batch_one<NP, TB, PASS_O1, TYPES>(B, eos, eps, citems, nf, nc, s, prepare);
  if (pass == PASS_PRED) return batch_one<NP, TB, PASS_PRED, TYPES>(B, eos, eps, citems, nf, nc, s, prepare);
  return batch_one<NP, TB, PASS_CORR, TYPES>(B, eos, eps, citems, nf, nc, s, prepare);
}

// fast: two phases, SG liquid then ideal gas, no THINC -- the kernels with the EOS types compiled in
static cudaError_t batch_launch(int np, int tb, int pass, const BatchParams& B, const ecg_eos* eos, double eps,
                                const BatchItem* citems, int nf, int nc, cudaStream_t s, bool prepare, bool fast) {
  // the batched workload's configuration: SG liquid, IG gas, van Leer everywhere
  constexpr int kSgIg = fast_code(eos_types_code<2>(ECG_EOS_SG, ECG_EOS_IG), ECG_LIM_VANLEER);
  if (np == 2 && fast) {
    if (tb == 64) return batch_tb<2, 64, kSgIg>(pass, B, eos, eps, citems, nf, nc, s, prepare);
    if (tb == 128) return batch_tb<2, 128, kSgIg>(pass, B, eos, eps, citems, nf, nc, s, prepare);
    return batch_tb<2, 256, kSgIg>(pass, B, eos, eps, citems, nf, nc, s, prepare);
  }
  if (np == 2) {
    if (tb == 64) return batch_tb<2, 64>(pass, B, eos, eps, citems, nf, nc, s, prepare);
    if (tb == 128) return batch_tb<2, 128>(pass, B, eos, eps, citems, nf, nc, s, prepare);
    return batch_tb<2, 256>(pass, B, eos, eps, citems, nf, nc, s, prepare);
  }
  if (tb == 64) return batch_tb<3, 64>(pass, B, eos, eps, citems, nf, nc, s, prepare);
  if (tb == 128) return batch_tb<3, 128>(pass, B, eos, eps, citems, nf, nc, s, prepare);
  return batch_tb<3, 256>(pass, B, eos, eps, citems, nf, nc, s, prepare);
}

}  // namespace ecg

using namespace ecg;

// The items of a part of the batch whose face fluxes fit the flux array: a pass runs its face kernel and its cell
// kernel piece by piece.
struct BatchPiece {
  int item0, nitems, citem0, ncitems;
};

struct ecg_batch {
  ecg_case c0;
  bool fast = false;  // kernels with the EOS types compiled in apply
  int ncases = 0, np = 2, order = 1, nstate = 0, nq = 0;
  int64_t total = 0;
  double eps = 0.;
  cudaStream_t stream = nullptr;
  std::vector<BatchCase> hcases;
  BatchCase* cases = nullptr;
  BatchScalars* scal = nullptr;
  double* state[2] = {nullptr, nullptr};
  double* half = nullptr;
  double* tmp = nullptr;
  DevStats* stats = nullptr;
  double* flux = nullptr;   // face fluxes, 3N + 4 per face
  int64_t nfaces = 0;       // faces it holds: all of them where memory allows
  BatchItem* items = nullptr;   // face items of the current tile, piece after piece
  BatchItem* citems = nullptr;  // cell items, piece after piece
  std::vector<BatchPiece> pieces;
  int tile = 128;
  int cur = 0;
  int newton_cap = 100;
  MlpDev* mlp = nullptr;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
};

namespace {

ecg_status bfail(cudaError_t e, const char* what) {
  set_error(std::string(what) + ": " + cudaGetErrorString(e));
  return ECG_ERR_CUDA;
}
#define BCUDA(call)                                    \
  do {                                                 \
    cudaError_t e_ = (call);                           \
    if (e_ != cudaSuccess) return bfail(e_, #call);    \
  } while (0)

void drop_graphs(ecg_batch* b) {
  for (int i = 0; i < 2; i++)
    if (b->graph[i]) {
      cudaGraphExecDestroy(b->graph[i]);
      b->graph[i] = nullptr;
    }
}

ecg_status upload_items(const std::vector<BatchItem>& it, BatchItem** out) {
  BCUDA(cudaMalloc(out, sizeof(BatchItem) * it.size()));
  BCUDA(cudaMemcpy(*out, it.data(), sizeof(BatchItem) * it.size(), cudaMemcpyHostToDevice));
  return ECG_OK;
}

// Lays the batch out in pieces of at most nfaces faces: runs of whole cases, a case that does not fit the rest of a
// piece cut at a multiple of CELL_THREADS cells.  The face at a cut belongs to both pieces (its flux and its wave
// speed are computed twice, to the same values).
ecg_status build_items(ecg_batch* b, int tile) {
  std::vector<BatchItem> it, ct;
  std::vector<BatchPiece> pieces;
  BatchPiece p{0, 0, 0, 0};
  int64_t used = 0;  // faces of the current piece
  auto close = [&] {
    p.nitems = (int)it.size() - p.item0;
    p.ncitems = (int)ct.size() - p.citem0;
    if (p.ncitems) pieces.push_back(p);
    p = {(int)it.size(), 0, (int)ct.size(), 0};
    used = 0;
  };
  for (int c = 0; c < b->ncases; c++) {
    const BatchCase& h = b->hcases[c];
    for (int s = 0; s < h.n;) {
      int64_t m = std::min<int64_t>(h.n - s, b->nfaces - used - 1);  // cells from s on whose faces fit
      if (m < h.n - s) m -= m % CELL_THREADS;
      if (m <= 0) {
        close();
        continue;
      }
      const int e = s + (int)m;
      const int64_t fbase = used - s;
      for (int f = s; f <= e; f += tile - 1) it.push_back({c, f, h.n, e, h.off, fbase});
      for (int g = s; g < e; g += CELL_THREADS) ct.push_back({c, g, h.n, e, h.off, fbase});
      used += m + 1;
      s = e;
    }
  }
  close();
  cudaFree(b->items);
  cudaFree(b->citems);
  b->items = b->citems = nullptr;
  b->pieces.clear();
  ecg_status st = upload_items(it, &b->items);
  if (st == ECG_OK) st = upload_items(ct, &b->citems);
  if (st == ECG_OK) b->pieces = pieces;
  return st;
}

// The flux array for all faces of the batch or, where they do not fit the GPU's free memory, for as many as leave as
// much again for the rest (a two-phase MUSCL batch: 21 doubles per cell and 10 per face).
cudaError_t alloc_flux(ecg_batch* b) {
  auto alloc = [&](int64_t faces) {
    const cudaError_t e = cudaMalloc(&b->flux, sizeof(double) * (size_t)(3 * b->np + 4) * (size_t)faces);
    if (e != cudaSuccess) {
      cudaGetLastError();  // the launches to come do not report it
      b->flux = nullptr;
    }
    b->nfaces = faces;
    return e;
  };
  int64_t faces = b->total + b->ncases;
  cudaError_t e = alloc(faces);
  if (e != cudaErrorMemoryAllocation) return e;
  constexpr int64_t kLeast = 1 << 14;
  while (e == cudaErrorMemoryAllocation && faces > 2 * kLeast) e = alloc(faces /= 2);
  if (e != cudaSuccess) return e;
  cudaFree(b->flux);
  return alloc(faces / 2);
}

ecg_status set_shape(ecg_batch* b, int tile) {
  if (tile != 64 && tile != 128 && tile != 256) {
    set_error("tile must be 64, 128 or 256 cells");
    return ECG_ERR_INVALID;
  }
  BatchParams B{};
  for (int pass : {PASS_O1, PASS_PRED, PASS_CORR})
    if ((pass == PASS_O1) == (b->order == 1))
      BCUDA(batch_launch(b->np, tile, pass, B, b->c0.eos, b->eps, nullptr, 0, 0, b->stream, true, b->fast));
  b->tile = tile;
  drop_graphs(b);
  return build_items(b, tile);
}

ecg_status launch_pass(ecg_batch* b, int pass, double* q, double* sn, double* out) {
  BatchParams B{};
  B.P.q = q;
  B.P.sn = sn;
  B.P.out = out;
  B.P.n = b->total;
  B.P.stats = b->stats;
  for (int i = 0; i < 4; i++) B.P.lim[i] = b->c0.limiter[i];
  B.P.newton_cap = b->newton_cap;
  set_thinc(B.P, b->c0);
  B.P.pt = b->c0.pt_relaxation;
  B.P.mlp = b->mlp;
  B.cases = b->cases;
  B.scal = b->scal;
  B.flux = b->flux;
  B.nfaces = b->nfaces;
  for (const BatchPiece& p : b->pieces) {
    B.items = b->items + p.item0;
    BCUDA(batch_launch(b->np, b->tile, pass, B, b->c0.eos, b->eps, b->citems + p.citem0, p.nitems, p.ncitems, b->stream,
                       false, b->fast));
  }
  return ECG_OK;
}

ecg_status launch_step(ecg_batch* b, int parity) {
  double* sn = b->state[parity];
  double* s1 = b->state[1 - parity];
  ecg_status s;
  if (b->order == 1) {
    s = launch_pass(b, PASS_O1, sn, sn, s1);
  } else {
    s = launch_pass(b, PASS_PRED, sn, sn, b->half);
    if (s == ECG_OK) s = launch_pass(b, PASS_CORR, b->half, sn, s1);
  }
  if (s != ECG_OK) return s;
  BCUDA(launch_chained(k_batch_finalize, dim3((b->ncases + 255) / 256), dim3(256), 0, b->stream, true, b->scal, b->cases,
                       b->ncases));
  return ECG_OK;
}

ecg_status advance(ecg_batch* b, int nsteps) {
  if (b->pieces.empty()) {  // no shape asked for yet
    const ecg_status s = set_shape(b, b->tile);
    if (s != ECG_OK) return s;
  }
  while (nsteps >= 2) {
    if (!b->graph[b->cur]) {
      cudaGraph_t g = nullptr;
      BCUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
      ecg_status s1 = launch_step(b, b->cur);
      ecg_status s2 = (s1 == ECG_OK) ? launch_step(b, 1 - b->cur) : s1;
      cudaError_t e = cudaStreamEndCapture(b->stream, &g);
      if (s2 != ECG_OK) {
        if (g) cudaGraphDestroy(g);
        return s2;
      }
      if (e != cudaSuccess) return bfail(e, "cudaStreamEndCapture");
      e = cudaGraphInstantiate(&b->graph[b->cur], g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return bfail(e, "cudaGraphInstantiate");
    }
    BCUDA(cudaGraphLaunch(b->graph[b->cur], b->stream));
    nsteps -= 2;
  }
  if (nsteps == 1) {
    ecg_status s = launch_step(b, b->cur);
    if (s != ECG_OK) return s;
    b->cur = 1 - b->cur;
  }
  return ECG_OK;
}

}  // namespace

extern "C" ecg_status ecg_batch_create(const ecg_case* cs, int32_t ncases, ecg_batch** out) {
  if (!cs || !out || ncases < 1) {
    set_error("bad argument");
    return ECG_ERR_INVALID;
  }
  *out = nullptr;
  const ecg_case& c0 = cs[0];
  if (c0.model != ECG_MODEL_KAPILA || c0.nphases < 2 || c0.nphases > 3 || c0.ptmu) {
    set_error("batched mode runs Kapila cases of 2 or 3 phases without p-T-mu relaxation");
    return ECG_ERR_UNSUPPORTED;
  }
  for (int c = 0; c < ncases; c++) {
    const ecg_case& x = cs[c];
    if (x.ncells[1] != 1 || x.ncells[2] != 1 || x.ncells[0] < 2) {
      set_error("batched mode runs 1D cases");
      return ECG_ERR_UNSUPPORTED;
    }
    if (x.ntransports != 0) {
      set_error("batched mode runs without passive transports");
      return ECG_ERR_UNSUPPORTED;
    }
    if (case_stretched(x)) {
      set_error("batched mode runs uniform meshes");
      return ECG_ERR_UNSUPPORTED;
    }
    if (x.bc[0] != ECG_BC_NONREFLECTING || x.bc[1] != ECG_BC_NONREFLECTING) {
      set_error("batched mode runs non-reflecting sides only");
      return ECG_ERR_UNSUPPORTED;
    }
    if (x.model != c0.model || x.nphases != c0.nphases || x.order != c0.order || x.alpha_null != c0.alpha_null ||
        std::memcmp(x.limiter, c0.limiter, sizeof(x.limiter)) != 0 || std::memcmp(x.eos, c0.eos, sizeof(x.eos)) != 0 ||
        x.pt_relaxation != c0.pt_relaxation) {
      set_error("all cases of a batch share model, phases, EOS, order, limiters and alphaNull");
      return ECG_ERR_INVALID;
    }
  }
  auto b = new ecg_batch();
  b->c0 = c0;
  b->fast = c0.nphases == 2 && c0.eos[0].type == ECG_EOS_SG && c0.eos[1].type == ECG_EOS_IG && !c0.pt_relaxation &&
            c0.order == 2 && c0.limiter[0] == ECG_LIM_VANLEER && c0.limiter[1] == ECG_LIM_VANLEER &&
            c0.limiter[2] == ECG_LIM_VANLEER && c0.limiter[3] == ECG_LIM_VANLEER;
  b->ncases = ncases;
  b->np = c0.nphases;
  b->order = c0.order;
  b->eps = c0.alpha_null ? 1.e-15 : 0.;
  b->nstate = 2 * b->np + 3;  // alpha_k, rho_k, p, u, E
  b->nq = b->nstate - 1;
  int64_t off = 0;
  for (int c = 0; c < ncases; c++) {
    const ecg_case& x = cs[c];
    BatchCase h{};
    h.off = off;
    h.n = x.ncells[0];
    double dX = x.length[0] / (double)x.ncells[0], dY = x.length[1] / (double)x.ncells[1],
           dZ = x.length[2] / (double)x.ncells[2];
    h.dx = dX;
    h.coefA = (dY * dZ) / (dX * dY * dZ);
    h.lcfl = std::min(1.e10, dX);
    h.cfl = x.cfl;
    b->hcases.push_back(h);
    off += h.n;
  }
  b->total = off;
  auto fail = [&](ecg_status s) {
    ecg_batch_destroy(b);
    return s;
  };
  cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) return fail(bfail(e, "cudaStreamCreate"));
  const size_t sb = sizeof(double) * (size_t)b->nstate * (size_t)b->total;
  for (int i = 0; i < 2; i++)
    if ((e = cudaMalloc(&b->state[i], sb)) != cudaSuccess) return fail(bfail(e, "cudaMalloc(state)"));
  if (b->order == 2 && (e = cudaMalloc(&b->half, sizeof(double) * (size_t)b->nq * b->total)) != cudaSuccess)
    return fail(bfail(e, "cudaMalloc(half)"));
  if ((e = cudaMalloc(&b->tmp, sizeof(double) * (size_t)b->total)) != cudaSuccess) return fail(bfail(e, "cudaMalloc"));
  if ((e = cudaMalloc(&b->cases, sizeof(BatchCase) * ncases)) != cudaSuccess) return fail(bfail(e, "cudaMalloc"));
  if ((e = cudaMalloc(&b->scal, sizeof(BatchScalars) * ncases)) != cudaSuccess) return fail(bfail(e, "cudaMalloc"));
  if ((e = cudaMalloc(&b->stats, sizeof(DevStats))) != cudaSuccess) return fail(bfail(e, "cudaMalloc"));
  if ((e = alloc_flux(b)) != cudaSuccess) return fail(bfail(e, "cudaMalloc(face fluxes)"));
  cudaMemcpy(b->cases, b->hcases.data(), sizeof(BatchCase) * ncases, cudaMemcpyHostToDevice);
  std::vector<BatchScalars> hs(ncases);
  double big = 1.e10;
  for (auto& s : hs) {
    s.dt = 1.e-15;
    s.t = 0.;
    std::memcpy(&s.dtmax_bits, &big, sizeof(double));
    s.it = 0;
  }
  cudaMemcpy(b->scal, hs.data(), sizeof(BatchScalars) * ncases, cudaMemcpyHostToDevice);
  // ordered before the batch's work, which all runs on its stream
  cudaMemsetAsync(b->stats, 0, sizeof(DevStats), b->stream);
  cudaMemsetAsync(b->state[0], 0, sb, b->stream);
  cudaMemsetAsync(b->state[1], 0, sb, b->stream);
  if ((e = cudaStreamSynchronize(b->stream)) != cudaSuccess) return fail(bfail(e, "create"));
  *out = b;
  return ECG_OK;
}

extern "C" void ecg_batch_destroy(ecg_batch* b) {
  if (!b) return;
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_graphs(b);
  cudaFree(b->state[0]);
  cudaFree(b->state[1]);
  cudaFree(b->half);
  cudaFree(b->tmp);
  cudaFree(b->cases);
  cudaFree(b->scal);
  cudaFree(b->stats);
  cudaFree(b->flux);
  cudaFree(b->items);
  cudaFree(b->citems);
  cudaFree(b->mlp);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

extern "C" int64_t ecg_batch_total_cells(const ecg_batch* b) { return b ? b->total : 0; }
extern "C" void* ecg_batch_stream(const ecg_batch* b) { return b ? (void*)b->stream : nullptr; }

extern "C" ecg_status ecg_batch_upload_prim(ecg_batch* b, const double* const* f, int64_t total) {
  if (!b || !f || total != b->total) {
    set_error("bad argument");
    return ECG_ERR_INVALID;
  }
  const int np = b->np;
  const size_t fb = sizeof(double) * (size_t)total;
  double* S = b->state[b->cur];
  for (int i = 0; i < 2 * np + 1; i++) BCUDA(cudaMemcpyAsync(S + (size_t)i * total, f[i], fb, cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(S + (size_t)(2 * np + 1) * total, f[2 * np + 1], fb, cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(S + (size_t)(2 * np + 2) * total, f[2 * np + 4], fb, cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaStreamSynchronize(b->stream));
  return ECG_OK;
}

namespace ecg {
__global__ void k_derived(const double* __restrict__ S, int64_t n, int np, int dim, ecg_eos e0, ecg_eos e1, ecg_eos e2,
                          double eps, double* pmix, double* T, double* Y);
}

extern "C" ecg_status ecg_batch_download_prim(ecg_batch* b, double* const* f, int64_t total) {
  if (!b || !f || total != b->total) {
    set_error("bad argument");
    return ECG_ERR_INVALID;
  }
  const int np = b->np;
  const size_t fb = sizeof(double) * (size_t)total;
  const double* S = b->state[b->cur];
  k_derived<<<(unsigned)((total + 255) / 256), 256, 0, b->stream>>>(S, total, np, 1, b->c0.eos[0], b->c0.eos[1],
                                                                     b->c0.eos[2], b->eps, b->tmp, nullptr, nullptr);
  BCUDA(cudaGetLastError());
  for (int i = 0; i < 2 * np; i++) BCUDA(cudaMemcpyAsync(f[i], S + (size_t)i * total, fb, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaMemcpyAsync(f[2 * np], b->tmp, fb, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaMemcpyAsync(f[2 * np + 1], S + (size_t)(2 * np + 1) * total, fb, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaMemcpyAsync(f[2 * np + 4], S + (size_t)(2 * np + 2) * total, fb, cudaMemcpyDeviceToHost, b->stream));
  std::memset(f[2 * np + 2], 0, fb);  // while the copies run
  std::memset(f[2 * np + 3], 0, fb);
  BCUDA(cudaStreamSynchronize(b->stream));
  return ECG_OK;
}

extern "C" ecg_status ecg_batch_step(ecg_batch* b, int32_t nsteps, double* dt, double* t, ecg_step_stats* stats) {
  if (!b || nsteps < 0) {
    set_error("bad argument");
    return ECG_ERR_INVALID;
  }
  const int nc = b->ncases;
  if (dt || t) {
    // the caller's per-case dt / t seed the device scalars
    std::vector<BatchScalars> hs(nc);
    BCUDA(cudaMemcpy(hs.data(), b->scal, sizeof(BatchScalars) * nc, cudaMemcpyDeviceToHost));
    for (int c = 0; c < nc; c++) {
      if (dt) hs[c].dt = dt[c];
      if (t) hs[c].t = t[c];
    }
    BCUDA(cudaMemcpyAsync(b->scal, hs.data(), sizeof(BatchScalars) * nc, cudaMemcpyHostToDevice, b->stream));
  }
  BCUDA(cudaMemsetAsync(b->stats, 0, sizeof(DevStats), b->stream));
  ecg_status s = advance(b, nsteps);
  if (s != ECG_OK) return s;
  DevStats ds{};
  BCUDA(cudaMemcpyAsync(&ds, b->stats, sizeof(ds), cudaMemcpyDeviceToHost, b->stream));
  if (dt || t) {
    std::vector<BatchScalars> hs(nc);
    BCUDA(cudaMemcpyAsync(hs.data(), b->scal, sizeof(BatchScalars) * nc, cudaMemcpyDeviceToHost, b->stream));
    BCUDA(cudaStreamSynchronize(b->stream));
    for (int c = 0; c < nc; c++) {
      if (dt) dt[c] = hs[c].dt;
      if (t) t[c] = hs[c].t;
    }
  }
  BCUDA(cudaStreamSynchronize(b->stream));
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->cell_updates = (int64_t)nsteps * b->total;
    stats->relax_calls = (int64_t)ds.relax_calls;
    stats->newton_evals = (int64_t)ds.newton_evals;
    stats->newton_fallback = (int64_t)ds.newton_fallback;
    stats->newton_max = (int64_t)ds.newton_max;
    stats->seeded = (int64_t)ds.seeded;
    stats->seed_rejected = (int64_t)ds.seed_rejected;
    stats->nonfinite_cells = (int64_t)ds.nonfinite;
    for (int i = 0; i < 16; i++) stats->newton_hist[i] = (int64_t)ds.hist[i];
  }
  return ECG_OK;
}

extern "C" ecg_status ecg_batch_set_seed_model(ecg_batch* b, const ecg_mlp* m) {
  if (!b) {
    set_error("null batch");
    return ECG_ERR_INVALID;
  }
  drop_graphs(b);
  if (!m) {
    cudaFree(b->mlp);
    b->mlp = nullptr;
    return ECG_OK;
  }
  return mlp_upload(m, b->np, false, &b->mlp, b->stream);
}

extern "C" ecg_status ecg_batch_set_shape(ecg_batch* b, int32_t tile, int32_t threads) {
  if (!b) {
    set_error("null batch");
    return ECG_ERR_INVALID;
  }
  if (tile == 0) {
    int32_t t2 = 0, th = 0;
    return ecg_batch_autotune(b, &t2, &th);
  }
  if (threads != 0 && threads != tile) {
    set_error("one thread per cell of a tile: threads must equal tile");
    return ECG_ERR_INVALID;
  }
  return set_shape(b, tile);
}

// Times two steps of every candidate tile on a copy of the current state and keeps the fastest.
extern "C" ecg_status ecg_batch_autotune(ecg_batch* b, int32_t* tile, int32_t* threads) {
  if (!b) {
    set_error("null batch");
    return ECG_ERR_INVALID;
  }
  const size_t sb = sizeof(double) * (size_t)b->nstate * (size_t)b->total;
  double* save = nullptr;
  BatchScalars* ssave = nullptr;
  BCUDA(cudaMalloc(&save, sb));
  cudaError_t e = cudaMalloc(&ssave, sizeof(BatchScalars) * b->ncases);
  if (e != cudaSuccess) {
    cudaFree(save);
    return bfail(e, "cudaMalloc");
  }
  const int cur0 = b->cur;
  cudaMemcpyAsync(save, b->state[cur0], sb, cudaMemcpyDeviceToDevice, b->stream);
  cudaMemcpyAsync(ssave, b->scal, sizeof(BatchScalars) * b->ncases, cudaMemcpyDeviceToDevice, b->stream);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int best = 128;
  float best_ms = 1e30f;
  ecg_status st = ECG_OK;
  for (int cand : {64, 128, 256}) {
    st = set_shape(b, cand);
    if (st != ECG_OK) break;
    b->cur = cur0;
    st = advance(b, 2);  // warm-up / graph capture
    if (st != ECG_OK) break;
    cudaMemcpyAsync(b->state[cur0], save, sb, cudaMemcpyDeviceToDevice, b->stream);
    cudaMemcpyAsync(b->scal, ssave, sizeof(BatchScalars) * b->ncases, cudaMemcpyDeviceToDevice, b->stream);
    b->cur = cur0;
    cudaEventRecord(e0, b->stream);
    st = advance(b, 2);
    cudaEventRecord(e1, b->stream);
    if (st != ECG_OK) break;
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best_ms) {
      best_ms = ms;
      best = cand;
    }
    cudaMemcpyAsync(b->state[cur0], save, sb, cudaMemcpyDeviceToDevice, b->stream);
    cudaMemcpyAsync(b->scal, ssave, sizeof(BatchScalars) * b->ncases, cudaMemcpyDeviceToDevice, b->stream);
  }
  cudaStreamSynchronize(b->stream);
  b->cur = cur0;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(save);
  cudaFree(ssave);
  cudaMemsetAsync(b->stats, 0, sizeof(DevStats), b->stream);
  if (st != ECG_OK) return st;
  st = set_shape(b, best);
  if (st != ECG_OK) return st;
  if (tile) *tile = best;
  if (threads) *threads = best;
  return ECG_OK;
}
