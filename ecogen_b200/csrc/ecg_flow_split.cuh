// Split form of an Euler or PTUEq step pass on 2D and 3D meshes: one face-flux kernel per axis, side by side,
// then one cell kernel (see ecg_kapila_split.cuh, whose tiles, staging and face arrays these kernels
// share; the reference lines of the physics stand at the functions they call, in ecg_euler.cuh and
// ecg_ptueq.cuh, which include this file).
//
// A model M supplies: Eos (its parameters), Side (a completed face side), NM mass fluxes, U (the plane of the
// first velocity; planes 0 .. U + DIM - 1 are the reconstructed fields, in the state's order), STORED (planes
// the first-order pass stages beyond those) and the functions
//   load      a side from staged cell rc (completed; `stored`: an interior face of the first-order pass)
//   extrapolate   a side from cell rc and its limited slopes, clamped and completed
//   wall_value / wall_flux   a symmetry side's buffer cell and its normal momentum flux
//   hllc      the flux through a face, masses, face-frame momentum, energy
//   update    U^n, time evolution and buildPrim of a cell from its accumulated fluxes
// The face arrays hold NM masses, DIM momenta and the energy.
//
// A case runs in this form when its limiter slots agree (cell_slopes' argument holds for any one limiter: the
// interface detector decides nothing, and each limiter is symmetric in its slopes) and it has neither THINC
// nor passive transports; otherwise the fused kernels run.  Why it is faster: the fused pass computed the
// faces and slopes of a tile's border twice, limited every slope twice and met a barrier per phase and axis.
// Measured on one B200 (mid-run states, per step): PTUEq 2048^2 1.93 -> 1.23 ms, Euler 2048^2 1.11 -> 0.80 ms (1.19 and 0.72 ms with the
// register budgets below);
// the same bits in every field.
#pragma once
#include "ecg_faces.cuh"

namespace ecg {

template <class MD, int DIM, int PASS>
struct FlowShape {
  static constexpr bool O2 = (PASS != PASS_O1);
  static constexpr int NSL = MD::U + DIM;
  static constexpr int NQ = NSL + (O2 ? 0 : MD::STORED);
  static constexpr int NFL = MD::NM + DIM + 1;
  static constexpr size_t staged_bytes() { return sizeof(double) * (size_t)FACE_RS * NQ; }
  static constexpr size_t smem_bytes() {
    return staged_bytes() + (O2 ? sizeof(double) * (size_t)FACE_LS * NSL : 0) + sizeof(uint64_t) + 128;
  }
};

// The faces normal to AX, one block per tile.  LIMC >= 0: the limiter, compiled in; -1: P.lim[0], read at run
// time.
template <class MD, int DIM, int AX, int PASS, int LIMC>
__global__ void __launch_bounds__(FACE_THREADS, DIM == 2 ? MD::FACE_MINB : 8)
    k_flow_faces(StepParams P, Geometry G, typename MD::Eos M, const __grid_constant__ FaceLaunch L) {
  using KS = FlowShape<MD, DIM, PASS>;
  constexpr bool O2 = KS::O2, isx = AX == 0;
  constexpr int NQ = KS::NQ, NSL = KS::NSL, U = MD::U, RS = FACE_RS, SS = FACE_LS, ax = AX, ob = isx ? 1 : 0;
  extern __shared__ unsigned char smem_raw[];
  double* sq = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);  // [NQ][RS]
  double* ssl = sq + (size_t)NQ * RS;                                                                      // [NSL][SS]
  const int done = *P.done;
  const int tid = threadIdx.x;
  const FacePlace B = face_place<AX>();
  const int f0 = B.f0, l0 = B.l0, third = B.third;
  constexpr int PS = isx ? 1 : FaceTile<1>::W;   // stride of a position along the axis
  constexpr int CL = isx ? FaceTile<0>::CP : 1;  // stride of a line, staged planes
  constexpr int SL = isx ? FaceTile<0>::LP : 1;  // ..., slope planes
  const int nax = G.n[ax];
  const int64_t nn = P.n;
  auto place = [&](int e, int len, int& line, int& pos) {
    if (isx) {
      line = e / len;
      pos = e - line * len;
    } else {
      line = e % FaceTile<1>::W;
      pos = e / FaceTile<1>::W;
    }
  };
  // ---- stage the cells from f0 - 2 of every line
  if (L.tma) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(sq + (size_t)NQ * RS + (O2 ? (size_t)SS * NSL : 0));
    if (tid == 0) mbar_init(bar, 1);
    __syncthreads();
    if (tid == 0) {
      mbar_expect_tx(bar, (uint32_t)KS::staged_bytes());
      const int ox = isx ? f0 - 2 : l0, oy = isx ? l0 : (ax == 1 ? f0 - 2 : third), oz = ax == 2 ? f0 - 2 : third;
      if (DIM == 3) tma_load_4d(sq, &L.q, bar, ox, oy, oz, 0);
      else tma_load_3d(sq, &L.q, bar, ox, oy, 0);
    }
    if (!mbar_wait_bounded(bar, 0, 1 << 22) && (tid & 31) == 0) atomicAdd(&P.stats->staging_timeouts, 1ull);
  } else {
    for (int e = tid; e < RS; e += FACE_THREADS) {
      int line, pos;
      place(e, FaceTile<0>::CP, line, pos);
      const int g = f0 - 2 + pos, lg = l0 + line;
      if (pos < (isx ? FaceTile<0>::TF : FaceTile<1>::TF) + 3 && g >= 0 && g < nax && lg < G.n[ob]) {
        const int cx = isx ? g : lg, cy = isx ? lg : (ax == 1 ? g : third), cz = ax == 2 ? g : third;
        const int64_t c = cx + (int64_t)G.n[0] * (cy + (int64_t)G.n[1] * cz);
        if (!ECG_IN_BOUNDS(P.stats, c, nn)) continue;
#pragma unroll
        for (int f = 0; f < NQ; f++) sq[f * RS + e] = P.q[(int64_t)f * nn + c];
      }
    }
  }
  if (done) return;  // tested here: the staging does not wait for it
  __syncthreads();
  // ---- limited slopes: cell f0 - 1 + s of every line, s in [0, TF]
  if (O2) {
    const int kind = LIMC >= 0 ? LIMC : P.lim[0];
    constexpr int nsl = isx ? FaceTile<0>::LS : FaceTile<1>::LS;
    const double *dcc = G.dcc[ax], *rdcc = G.rdcc[ax];
    for (int e = tid; e < nsl; e += FACE_THREADS) {
      int line, s;
      place(e, FaceTile<0>::LP, line, s);
      const int c = f0 - 1 + s;
      if (c < 0 || c >= nax || l0 + line >= G.n[ob]) continue;
      const int rc = line * CL + (s + 1) * PS;
      if (c == 0 || c == nax - 1) {
        // no face beyond: every limited slope is zero, except the velocity along the axis at a symmetry side,
        // whose slope there is u over the centre-to-face coordinate (BoundCondWallO2Cartesian::computeSlopes
        // :84-108)
#pragma unroll
        for (int f = 0; f < NSL; f++) ssl[f * SS + e] = 0.;
        const int sd = c == 0 ? 0 : 1;
        const double wd = G.wslope[2 * ax + sd];
        if (G.bc[2 * ax + sd] == ECG_BC_SYMMETRY && fabs(wd) > 1.e-8) {
          const double* su = sq + (U + ax) * RS;
          const double so = sd ? ndiv(su[rc] - su[rc - PS], dcc[c - 1]) : ndiv(su[rc + PS] - su[rc], dcc[c]);
          ssl[(U + ax) * SS + e] = limiter(kind, ndiv(su[rc], wd), so);
        }
        continue;
      }
      const double dm = dcc[c - 1], rm = rdcc[c - 1], dp = dcc[c], rp = rdcc[c];
#pragma unroll
      for (int f = 0; f < NSL; f++) {
        const double v = sq[f * RS + rc];
        ssl[f * SS + e] = limiter(kind, cdiv(v - sq[f * RS + rc - PS], dm, rm), cdiv(sq[f * RS + rc + PS] - v, dp, rp));
      }
    }
    __syncthreads();
  }
  // ---- one face per thread
  double wmax = wave_none(G.stretched);
  {
    int line, fl;
    place(tid, FaceTile<0>::TF, line, fl);
    const int f = f0 + fl, lg = l0 + line;
    auto lcfl = [&](int g) {
      return G.stretched ? cell_lcfl(G, isx ? g : lg, isx ? lg : (ax == 1 ? g : third), ax == 2 ? g : third) : G.lcfl;
    };
    const int rl = line * CL + (fl + 1) * PS, rr = rl + PS;  // the cells on its two sides
    const int el = line * SL + fl * PS;                      // the left one's limited slopes
    if (f <= nax && lg < G.n[ob] && ECG_IN_BOUNDS(P.stats, rl, RS) && ECG_IN_BOUNDS(P.stats, rr, RS)) {
      constexpr int pn = ax, p1 = isx ? 1 : 0, p2 = ax == 2 ? 1 : 2;  // normal and transverse velocities
      double Fm[MD::NM], Fn[3], FE;
      typename MD::Side A, C;
      if (f == 0 || f == nax) {
        const int sd = f == 0 ? 0 : 1, rc = sd == 0 ? rr : rl;
        const double lc = lcfl(sd == 0 ? 0 : nax - 1);
        if (G.bc[2 * ax + sd] == ECG_BC_SYMMETRY) {
          MD::template wall<DIM, O2>(M, sq, RS, rc, ssl, SS, sd == 0 ? el + PS : el, ax, pn, p1, p2, G.wdist[2 * ax + sd], A);
          if (sd == 0) A.ul[0] = -A.ul[0];
          const double sL = dmin(A.ul[0] - A.c, -A.ul[0] - A.c);
          wave_add(wmax, G.stretched, sL, lc);
#pragma unroll
          for (int k = 0; k < MD::NM; k++) Fm[k] = 0.;
          Fn[0] = MD::wall_flux(A, sL);
          Fn[1] = Fn[2] = FE = 0.;
        } else {  // HLLC(cell, cell) in the side's frame
          MD::template load<DIM>(M, sq, RS, rc, ax, pn, p1, p2, false, A);
          if (sd == 0) A.ul[0] = -A.ul[0];
          MD::hllc(A, A, G.stretched, lc, lc, wmax, Fm, Fn, FE);
        }
        if (sd == 0) Fn[0] = -Fn[0];
      } else {
        const int gl = f - 1;
        if (O2) {
          MD::template extrapolate<DIM>(M, sq, RS, rl, ssl, SS, el, ax, pn, p1, p2, G.dfl[ax][gl], 1., A);
          MD::template extrapolate<DIM>(M, sq, RS, rr, ssl, SS, el + PS, ax, pn, p1, p2, G.dfr[ax][gl], -1., C);
        } else {
          MD::template load<DIM>(M, sq, RS, rl, ax, pn, p1, p2, true, A);
          MD::template load<DIM>(M, sq, RS, rr, ax, pn, p1, p2, true, C);
        }
        MD::hllc(A, C, G.stretched, lcfl(gl), lcfl(gl + 1), wmax, Fm, Fn, FE);
      }
      const int64_t nfa = split_nfaces(G.n, ax);
      const int64_t fid = split_fid(G.n, ax, f, lg, isx ? lg : third, third);
      if (ECG_IN_BOUNDS(P.stats, fid, nfa)) {
        double* out = L.flux + fid;
#pragma unroll
        for (int k = 0; k < MD::NM; k++) out[(int64_t)k * nfa] = Fm[k];
        out[(int64_t)(MD::NM + pn) * nfa] = Fn[0];
        out[(int64_t)(MD::NM + p1) * nfa] = Fn[1];
        if (DIM > 2) out[(int64_t)(MD::NM + p2) * nfa] = Fn[2];
        out[(int64_t)(MD::NM + DIM) * nfa] = FE;
      }
    }
  }
  // ---- dtMax: block reduction of the wave speeds, one atomic per block
  __shared__ double red[FACE_THREADS / 32];
  double v = wmax;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < FACE_THREADS / 32; w++) v = dmax(v, red[w]);
    atomic_min_pos_double(P.dtmax_bits, wave_dtmax(v, G.stretched, G.lcfl));
  }
}

// One thread per cell: its faces' fluxes in the reference's order (axis by axis the left face added, the right
// one subtracted; then the domain sides), then the model's update.
template <class MD, int DIM, int PASS>
__global__ void __launch_bounds__(128, DIM == 2 ? MD::CELL_MINB : 8)
    k_flow_cells(StepParams P, Geometry G, typename MD::Eos M, FaceArrays FA) {
  constexpr int NFL = MD::NM + DIM + 1;
  const int done = *P.done;
  const int64_t nn = P.n;
  const int64_t cell = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (cell >= nn) return;
  // copied ahead: the last axis' two face fluxes and the time-n state (measured, per step at 2048^2: Euler 717 ->
  // 697 us, PTUEq 1188 -> 1141 us; the kernel waited for loads 10.7 of 16.9 cycles between issues)
  constexpr int LA = DIM - 1, NS = MD::U + DIM + 1;
  __shared__ double stage[2 * NFL + NS][128];
  const int g[3] = {(int)(cell % G.n[0]), (int)((cell / G.n[0]) % G.n[1]), (int)(cell / ((int64_t)G.n[0] * G.n[1]))};
  {
    const int64_t nfa = split_nfaces(G.n, LA);
    const double* lo = FA.flux[LA] + split_fid(G.n, LA, g[LA], g[0], g[1], g[2]);
    const double* hi = FA.flux[LA] + split_fid(G.n, LA, g[LA] + 1, g[0], g[1], g[2]);
#pragma unroll
    for (int i = 0; i < NFL; i++) {
      cell_copy(&stage[i][threadIdx.x], lo + (int64_t)i * nfa);
      cell_copy(&stage[NFL + i][threadIdx.x], hi + (int64_t)i * nfa);
    }
#pragma unroll
    for (int i = 0; i < NS; i++) cell_copy(&stage[2 * NFL + i][threadIdx.x], P.sn + (int64_t)i * nn + cell);
  }
  double acc[NFL];
#pragma unroll
  for (int i = 0; i < NFL; i++) acc[i] = 0.;
#pragma unroll
  for (int ax = 0; ax < DIM; ax++) {
    const int64_t nfa = split_nfaces(G.n, ax);
    const double cA = cell_coefA(G, ax, g[0], g[1], g[2]);
    const int64_t fl = split_fid(G.n, ax, g[ax], g[0], g[1], g[2]), fr = split_fid(G.n, ax, g[ax] + 1, g[0], g[1], g[2]);
    if (!ECG_IN_BOUNDS(P.stats, fl, nfa) || !ECG_IN_BOUNDS(P.stats, fr, nfa)) return;  // (bounds-checked builds)
    double a[NFL], b[NFL];
    if (ax == LA) cell_copies_wait();
#pragma unroll
    for (int i = 0; i < NFL; i++) {
      a[i] = ax == LA ? stage[i][threadIdx.x] : FA.flux[ax][(int64_t)i * nfa + fl];
      b[i] = ax == LA ? stage[NFL + i][threadIdx.x] : FA.flux[ax][(int64_t)i * nfa + fr];
    }
    if (g[ax] >= 1) {
#pragma unroll
      for (int i = 0; i < NFL; i++) acc[i] += cA * a[i];
    }
    if (g[ax] + 1 <= G.n[ax] - 1) {
#pragma unroll
      for (int i = 0; i < NFL; i++) acc[i] -= cA * b[i];
    }
  }
#pragma unroll
  for (int bf = 0; bf < 2 * DIM; bf++) {
    const int ax = bf >> 1;
    const bool neg = (bf & 1) == 0;
    if (neg ? (g[ax] != 0) : (g[ax] != G.n[ax] - 1)) continue;
    const int64_t nfa = split_nfaces(G.n, ax), fid = split_fid(G.n, ax, neg ? 0 : G.n[ax], g[0], g[1], g[2]);
    const double cA = cell_coefA(G, ax, g[0], g[1], g[2]);
#pragma unroll
    for (int i = 0; i < NFL; i++) acc[i] -= cA * FA.flux[ax][(int64_t)i * nfa + fid];
  }
  if (done) return;
  MD::template update<DIM, PASS>(P, M, nn, cell, acc, &stage[2 * NFL][threadIdx.x], 128);
}

template <class MD, int DIM, int AX, int PASS, int LIMC>
cudaError_t launch_flow_faces(const StepParams& P, const Geometry& G, const typename MD::Eos& M, cudaStream_t s,
                              bool prepare) {
  auto kern = k_flow_faces<MD, DIM, AX, PASS, LIMC>;
  const size_t sm = FlowShape<MD, DIM, PASS>::smem_bytes();
  if (prepare) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  const FaceLaunch L = face_launch<AX>(P, false);
  kern<<<face_grid<AX>(G.n), FACE_THREADS, sm, s>>>(P, G, M, L);
  return cudaGetLastError();
}

template <class MD, int DIM, int PASS, int LIMC>
cudaError_t launch_flow(const StepParams& P, const Geometry& G, const typename MD::Eos& M, cudaStream_t s, bool prepare) {
  const cudaError_t e = face_axes<DIM>(P, s, prepare, [&](auto ax, cudaStream_t sa) {
    return launch_flow_faces<MD, DIM, decltype(ax)::value, PASS, LIMC>(P, G, M, sa, prepare);
  });
  if (e != cudaSuccess || prepare) return e;
  FaceArrays FA{};
  for (int ax = 0; ax < DIM; ax++) FA.flux[ax] = P.flux[ax];
  const cudaError_t ee = end_begin(P, s);
  if (ee != cudaSuccess) return ee;
  k_flow_cells<MD, DIM, PASS><<<(unsigned)((P.n + 127) / 128), 128, 0, s>>>(P, G, M, FA);
  const cudaError_t ec = cudaGetLastError();
  return ec == cudaSuccess ? end_join(P, s) : ec;
}

// One pass of a model in split form (the caller has checked P.flux).
template <class MD, int DIM>
cudaError_t flow_pass(int pass, const StepParams& P, const Geometry& G, const typename MD::Eos& M, cudaStream_t s,
                      bool prepare) {
  // the limiter of the shipped workloads, compiled in (measured at 2048^2, us per call, limiter at run time / compiled
  // in: PTUEq 7446 / 7093, Euler 6037 / 5795); the others are read at run time by the same kernel
  const bool vl = P.lim[0] == ECG_LIM_VANLEER;
  if (pass == PASS_O1) return launch_flow<MD, DIM, PASS_O1, -1>(P, G, M, s, prepare);
  if (pass == PASS_PRED)
    return vl ? launch_flow<MD, DIM, PASS_PRED, ECG_LIM_VANLEER>(P, G, M, s, prepare)
              : launch_flow<MD, DIM, PASS_PRED, -1>(P, G, M, s, prepare);
  return vl ? launch_flow<MD, DIM, PASS_CORR, ECG_LIM_VANLEER>(P, G, M, s, prepare)
            : launch_flow<MD, DIM, PASS_CORR, -1>(P, G, M, s, prepare);
}

}  // namespace ecg
