// Split form of a Kapila step pass for 2D and 3D meshes: one face-flux kernel per axis, side by side, then
// one cell kernel.
//
// The fused pass (ecg_kapila_kernel.cuh) stages a tile per axis, computes its faces and accumulates
// them in one kernel: every block runs the whole pass (both axes' slopes, reconstructions and HLLC
// solves, then the relaxation) with a barrier after each phase, so warps whose faces took the cheap
// HLLC branch wait at the barrier for the ones sampling a star state, and the kernel's code (one copy
// of the face work per axis) is larger than the instruction cache.  The split form trades HBM
// traffic, of which the pass uses a few percent, for latency:
//   k_kapila_faces       one thread per face: stage the cells and the slopes of a block (a barrier after each), then
//                        reconstruct both sides and solve HLLC exactly as the fused pass does, including the domain sides (non-reflecting: HLLC(cell, cell) in
//                        the side's frame; symmetry: the reflecting flux of the MUSCL buffer cell), and
//                        store the face flux (3N + d + 3 doubles) in a face array of the axis;
//                        min-reduce lCFL/|s| into dtMax;
//   k_kapila_cells       one thread per cell, no barrier but the counters' (in 2D each thread copies the last
//                        axis' fluxes, u and E ahead into shared slots of its own): add and subtract the stored fluxes in the reference's face order (X faces, Y faces,
//                        Z faces, then sides Xm, Xp, Ym, Yp, Zm, Zp, src/Meshes/MeshCartesian.cpp:281-557)
//                        with the same non-conservative terms, then buildPrim, relaxations, energy
//                        correction and store (kapila_rebuild / kapila_finish).
// Every flux is computed once, by the same device functions in the same operation order, and each cell
// accumulates the same values in the same order, so the split and fused forms give identical bits.
//
// Face arrays: per axis, structure of arrays, NFL components of nfaces(AX) doubles (split_fid, ecg_faces.cuh).
#pragma once
#include "ecg_faces.cuh"
#include "ecg_kapila_kernel.cuh"

namespace ecg {

template <int NP, int DIM, int PASS, int TYPES>
struct FaceKernelShape {
  using FL = Fields<NP, DIM>;
  static constexpr bool O2 = (PASS != PASS_O1);
  // one limiter compiled in: limited slopes per cell (cell_slopes), no interface detector
  static constexpr bool LSL = O2 && code_limiter(TYPES) >= 0;
  static constexpr int NA0 = (PASS == PASS_CORR && !LSL) ? 1 : 0;  // separate time-n alpha_0 plane
  static constexpr int RS = FACE_RS;
  static constexpr int SS = LSL ? FACE_LS : FACE_SS;               // one slope plane
  static constexpr size_t staged_bytes() { return sizeof(double) * (size_t)RS * (FL::NQ + NA0); }
  // staged planes, slope planes, the staging mbarrier, and room to align the base to 128 bytes
  static constexpr size_t smem_bytes() {
    return staged_bytes() + (O2 ? sizeof(double) * (size_t)SS * FL::NSL : 0) + sizeof(uint64_t) + 128;
  }
};

// Resident blocks per SM asked of the face and cell kernels (registers 65536 / (128 x MINB)).  Measured on one
// B200 (per-kernel CUDA events, mid-run states; X / Y faces, cells of the predictor): 2D two-phase 2048^2 face
// kernels at 7 blocks 304 / 287 us, at 8 (64 registers) 288 / 270, at 9 302 / 281; cell kernel at 5 blocks 360 us,
// at 6 (80 registers) 346, but 26 us against 23 on 191 x 103 cells, where the spills of the Newton loop are not
// hidden; at 4 384 us.  3D three-phase 256^3 face kernels at 5 blocks 1.83 / 1.65 ms, at 6 (80 registers) 1.82 /
// 1.64, at 7 1.94 / 1.70; cell kernel at 5 2.26 ms, at 6 3.50, at 4 2.45.
#ifndef ECG_FACE_MINB_2D
#define ECG_FACE_MINB_2D 8
#endif
#ifndef ECG_FACE_MINB_3D
#define ECG_FACE_MINB_3D 6
#endif
#ifndef ECG_CELL_MINB
#define ECG_CELL_MINB 5
#endif
// The cell kernels with the learned pressure seed: the network's MMA fragments and features need
// registers (at 96 the seeded kernels spilled about 600 B).  Measured (seeded arm, CUDA events, 100
// steps): 3D cavity 256^3 at 5 blocks per SM 684.8 M cell-updates/s, at 4 (128 registers) 708.8 M, at 3
// 681.9 M; 2D shock-bubble 2048^2 1668.8 M, 1851.1 M and 1700.3 M.
#ifndef ECG_CELL_SEED_MINB
#define ECG_CELL_SEED_MINB 4
#endif
// The p-T-mu cell kernels run one warp per block: their cells take very different numbers of Newton
// iterations, and in 4-warp blocks the warps that finish first waited at the block's counter reduction
// for the slowest one (barrier stalls were 5.6 of 12.4 cycles between issues on the 1024^2 expansion),
// holding their slots; a one-warp block frees its slot for the next block as soon as it is done.
// 24 such blocks per SM (80 registers, no spill in the loops): measured on the 1024^2 expansion, cell kernel at 16
// blocks 0.392 ms, at 20 0.395, at 24 0.360, at 32 0.373.
#ifndef ECG_CELL_PTMU_THREADS
#define ECG_CELL_PTMU_THREADS 32
#endif
#ifndef ECG_CELL_PTMU_MINB
#define ECG_CELL_PTMU_MINB (768 / ECG_CELL_PTMU_THREADS)
#endif
constexpr int CELL_THREADS = 128;
__host__ __device__ constexpr int cell_threads(bool ptmu) { return ptmu ? ECG_CELL_PTMU_THREADS : CELL_THREADS; }

// A face of a block: its position along the axis, line and third coordinate, the staged cell left of it, that
// cell's limited slopes (or the face slope left of it), and whether no staged pressure is below a floor.
struct FaceAt {
  int f, lg, third, rl, el;
  bool pone;
};

// CFL length of the cell at position g of the line.
template <int AX>
__device__ __forceinline__ double face_lcfl(const Geometry& G, int g, int lg, int third) {
  return cell_lcfl(G, AX == 0 ? g : lg, AX == 0 ? lg : (AX == 1 ? g : third), AX == 2 ? g : third);
}

// Face-frame velocity (normal, transverse) of a global one; neg: the frame of a minus side.
template <int AX>
__device__ __forceinline__ void face_frame(const double u[3], bool neg, double l[3]) {
  l[0] = neg ? -u[AX] : u[AX];
  l[1] = AX == 0 ? u[1] : u[0];
  l[2] = AX == 2 ? u[1] : u[2];
}

template <int NP, int DIM, int AX>
__device__ __forceinline__ void store_face(const StepParams& P, const Geometry& G, double* flux, int f, int lg,
                                           int third, const double Fn[3], const Flux<NP>& F) {
  const int64_t nfa = split_nfaces(G.n, AX);
  const int64_t fid = split_fid(G.n, AX, f, lg, AX == 0 ? lg : third, third);
  if (!ECG_IN_BOUNDS(P.stats, fid, nfa)) return;
  constexpr int p1 = AX == 0 ? 1 : 0, p2 = AX == 2 ? 1 : 2;  // planes of the transverse momenta
  double* out = flux + fid;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    out[(int64_t)k * nfa] = F.a[k];
    out[(int64_t)(NP + k) * nfa] = F.m[k];
    out[(int64_t)(2 * NP + k) * nfa] = F.en[k];
  }
  out[(int64_t)(3 * NP + AX) * nfa] = Fn[0];
  out[(int64_t)(3 * NP + p1) * nfa] = Fn[1];
  if (DIM > 2) out[(int64_t)(3 * NP + p2) * nfa] = Fn[2];
  out[(int64_t)(3 * NP + DIM) * nfa] = F.E;
  out[(int64_t)(3 * NP + DIM + 1) * nfa] = F.sM;
  out[(int64_t)(3 * NP + DIM + 2) * nfa] = F.uStar;
}

// The two sides of an internal face, from the block's staged planes; FULFILL: their closure too.
template <int NP, int DIM, int AX, int PASS, int TYPES, bool FULFILL>
__device__ __forceinline__ void face_sides(const StepParams& P, const Geometry& G, const Model<NP>& M, const double* sq,
                                           const FaceAt& A, Thermo<NP>& tl, double ul[3], Thermo<NP>& tr,
                                           double ur[3]) {
  using KS = FaceKernelShape<NP, DIM, PASS, TYPES>;
  using FL = Fields<NP, DIM>;
  constexpr int RS = KS::RS, SS = KS::SS, PS = AX == 0 ? 1 : FaceTile<1>::W;
  constexpr int p1 = AX == 0 ? 1 : 0, p2 = AX == 2 ? 1 : 2;
  const double* a0 = KS::NA0 ? sq + (size_t)FL::NQ * RS : sq;  // time-n alpha_0 plane
  const double* ssl = sq + (size_t)(FL::NQ + KS::NA0) * RS;
  const int gl = A.f - 1, rl = A.rl, rr = rl + PS, nax = G.n[AX];
  if (KS::LSL) {
    extrapolate_side<NP, DIM, FULFILL>(M, sq, RS, rl, ssl, SS, A.el, AX, p1, p2, G.dfl[AX][gl], 1., A.pone, tl, ul);
    extrapolate_side<NP, DIM, FULFILL>(M, sq, RS, rr, ssl, SS, A.el + PS, AX, p1, p2, G.dfr[AX][gl], -1., A.pone, tr, ur);
    return;
  }
  double ug[3], vg[3];
  if (!KS::O2) {
    cell_thermo<NP, DIM, FULFILL>(M, sq, RS, rl, tl, ug);
    cell_thermo<NP, DIM, FULFILL>(M, sq, RS, rr, tr, vg);
  } else {
    const int f1 = A.el + PS;  // this face
    const bool hasL = (gl - 1 >= 0), hasR = (gl + 2 < nax);
    // beyond a symmetry side the opposite slope is the side's and alphaCellAfterOppositeSide is the
    // cell's own time-n alpha (CellO2Cartesian::computeLocalSlopes :68-71); a non-reflecting side
    // has neither
    const bool wL = !hasL && G.bc[2 * AX] == ECG_BC_SYMMETRY;
    const bool wR = !hasR && G.bc[2 * AX + 1] == ECG_BC_SYMMETRY;
    const int f2l = (hasL || wL) ? A.el : -1;           // face (gl-1, gl)
    const int f2r = (hasR || wR) ? A.el + 2 * PS : -1;  // face (gl+1, gl+2)
    const double aL = sq[FL::A * RS + rl], aR = sq[FL::A * RS + rr];
    const double aLL = hasL ? a0[rl - PS] : (wL ? a0[rl] : 0.);
    const double aRR = hasR ? a0[rr + PS] : (wR ? a0[rr] : 0.);
    constexpr bool kThinc = (TYPES == EOS_DYNAMIC);
    constexpr int kLim = code_limiter(TYPES);
    reconstruct_side<NP, DIM, kThinc, kLim, FULFILL>(M, P, sq, RS, rl, ssl, SS, f1, f2l, aL, aR, aLL, G.dfl[AX][gl], 1.,
                                                     tl, ug);
    reconstruct_side<NP, DIM, kThinc, kLim, FULFILL>(M, P, sq, RS, rr, ssl, SS, f1, f2r, aR, aL, aRR, G.dfr[AX][gl],
                                                     -1., tr, vg);
  }
  face_frame<AX>(ug, false, ul);
  face_frame<AX>(vg, false, ur);
}

// Any face of a block, domain sides included, solved by fulfill and hllc and stored; returns its wave value
// (wave_add).  Out of line: the kernel holds the ordinary face only, and calls this for symmetry sides and
// for the faces hllc_quick leaves.
template <int NP, int DIM, int AX, int PASS, int TYPES>
static __device__ __noinline__ double face_general(const StepParams& P, const Geometry& G, const Model<NP>& M0,
                                                   double* flux, const double* sq, const FaceAt A) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);
  using KS = FaceKernelShape<NP, DIM, PASS, TYPES>;
  using FL = Fields<NP, DIM>;
  constexpr bool O2 = KS::O2;
  constexpr int RS = KS::RS, SS = KS::SS, PS = AX == 0 ? 1 : FaceTile<1>::W;
  const double* a0 = KS::NA0 ? sq + (size_t)FL::NQ * RS : sq;
  const double* ssl = sq + (size_t)(FL::NQ + KS::NA0) * RS;
  const int nax = G.n[AX];
  double wmax = wave_none(G.stretched), Fn[3];
  Flux<NP> F;
  if (A.f == 0 || A.f == nax) {
    // a side: non-reflecting HLLC(cell, cell) in the side's frame (BoundCondNonReflecting::
    // solveRiemannBoundary src/BoundConds/BoundCondNonReflecting.cpp:62), or a symmetry side's
    // reflecting flux (ModUEq::solveRiemannWall src/Models/UEq/ModUEq.cpp:452) of the buffer cell,
    // MUSCL-extrapolated towards the side (BoundCondWallO2Cartesian::solveRiemann :111-141)
    const int sd = (A.f == 0) ? 0 : 1;
    const bool neg = sd == 0;
    const int rc = sd == 0 ? A.rl + PS : A.rl;
    const double lc = face_lcfl<AX>(G, sd == 0 ? 0 : nax - 1, A.lg, A.third);
    Thermo<NP> t;
    double ug[3], ul[3];
    if (G.bc[2 * AX + sd] == ECG_BC_SYMMETRY) {
      if (KS::LSL) {
        wall_side_limited<NP, DIM>(M, sq, RS, rc, ssl, SS, sd == 0 ? A.el + PS : A.el, G.wdist[2 * AX + sd], t, ug);
      } else if (O2) {
        wall_side<NP, DIM>(M, P.lim, sq, RS, rc, ssl, SS, A.el + PS, sd == 0 ? A.el + 2 * PS : A.el, a0[rc],
                           G.wdist[2 * AX + sd], t, ug);
      } else {
        cell_thermo<NP, DIM>(M, sq, RS, rc, t, ug);
      }
      face_frame<AX>(ug, neg, ul);
      const double pstar = wall_pstar<NP>(t, ul, G.stretched, lc, wmax);
#pragma unroll
      for (int k = 0; k < NP; k++) F.a[k] = F.m[k] = F.en[k] = 0.;
      F.E = 0.;
      F.sM = 0.;
      F.uStar = 0.;
      Fn[0] = pstar;
      Fn[1] = 0.;
      Fn[2] = 0.;
    } else {
      cell_thermo<NP, DIM>(M, sq, RS, rc, t, ug);
      face_frame<AX>(ug, neg, ul);
      hllc<NP>(M, t, ul, t, ul, G.stretched, lc, lc, wmax, Fn, F);
    }
    if (neg) Fn[0] = -Fn[0];
  } else {
    Thermo<NP> tl, tr;
    double ul[3], ur[3];
    face_sides<NP, DIM, AX, PASS, TYPES, true>(P, G, M, sq, A, tl, ul, tr, ur);
    hllc<NP, O2>(M, tl, ul, tr, ur, G.stretched, face_lcfl<AX>(G, A.f - 1, A.lg, A.third),
                 face_lcfl<AX>(G, A.f, A.lg, A.third), wmax, Fn, F);
  }
  store_face<NP, DIM, AX>(P, G, flux, A.f, A.lg, A.third, Fn, F);
  return wmax;
}

// The faces normal to AX, one block per tile.  The transverse velocities enter without the sign changes of
// the face frames (src/Meshes/MeshCartesian.cpp:281-557); they only occur squared and as factors of their own
// momentum flux, whose sign changes back.
template <int NP, int DIM, int AX, int PASS, int TYPES>
__global__ void __launch_bounds__(FACE_THREADS, DIM == 2 ? ECG_FACE_MINB_2D : ECG_FACE_MINB_3D)
    k_kapila_faces(const __grid_constant__ StepParams P, const __grid_constant__ Geometry G,
                   const __grid_constant__ Model<NP> M0, const __grid_constant__ FaceLaunch L) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);
  using KS = FaceKernelShape<NP, DIM, PASS, TYPES>;
  using FL = Fields<NP, DIM>;
  constexpr bool O2 = KS::O2, LSL = KS::LSL;
  constexpr int RS = KS::RS, SS = KS::SS, ax = AX;
  extern __shared__ unsigned char smem_raw[];
  double* smem = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  double* sq = smem;                                // [NQ][RS]
  double* sa0 = sq + (size_t)FL::NQ * RS;           // [NA0][RS]
  double* ssl = sa0 + (size_t)KS::NA0 * RS;         // [NSL][SS]
  const double* a0 = KS::NA0 ? sa0 : sq;            // time-n alpha_0 plane
  const int done = *P.done;
  const int tid = threadIdx.x;
  constexpr bool isx = ax == 0;
  const FacePlace B = face_place<AX>();
  const int f0 = B.f0, l0 = B.l0, third = B.third;
  // tile: TF faces per line; a staged plane and a slope plane as [line][position] (X) or [position][line]
  constexpr int TF = isx ? FaceTile<0>::TF : FaceTile<1>::TF;
  constexpr int PS = isx ? 1 : FaceTile<1>::W;          // stride of a position (staged planes and slope planes)
  constexpr int CL = isx ? FaceTile<0>::CP : 1;         // stride of a line, staged planes
  constexpr int SL = isx ? (LSL ? FaceTile<0>::LP : FaceTile<0>::SP) : 1;  // ..., slope planes
  constexpr int nsl = LSL ? (isx ? FaceTile<0>::LS : FaceTile<1>::LS) : (isx ? FaceTile<0>::SS : FaceTile<1>::SS);
  const int nax = G.n[ax];
  constexpr int ob = isx ? 1 : 0;                       // the lines' axis
  const int64_t nn = P.n;
  // (line, position) of entry e of a plane whose lines hold `len` entries
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
    // one tensor copy of the box (x, y[, z], field) for all primitive fields, one for the time-n
    // alpha_0 plane; cells outside the mesh arrive as zeros
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + KS::staged_bytes() / sizeof(double) +
                                                (O2 ? (size_t)SS * FL::NSL : 0));
    if (tid == 0) mbar_init(bar, 1);
    __syncthreads();
    if (tid == 0) {
      mbar_expect_tx(bar, (uint32_t)KS::staged_bytes());
      // box origin along x, y, z
      const int ox = isx ? f0 - 2 : l0, oy = isx ? l0 : (ax == 1 ? f0 - 2 : third), oz = ax == 2 ? f0 - 2 : third;
      if (DIM == 3) {
        tma_load_4d(sq, &L.q, bar, ox, oy, oz, 0);
        if (KS::NA0) tma_load_4d(sa0, &L.a0, bar, ox, oy, oz, FL::A);
      } else {
        tma_load_3d(sq, &L.q, bar, ox, oy, 0);
        if (KS::NA0) tma_load_3d(sa0, &L.a0, bar, ox, oy, FL::A);
      }
    }
    // bounded wait; a copy that never lands is reported to the host (the step then fails)
    if (!mbar_wait_bounded(bar, 0, 1 << 22) && (tid & 31) == 0) atomicAdd(&P.stats->staging_timeouts, 1ull);
  } else {
    for (int e = tid; e < RS; e += FACE_THREADS) {
      int line, pos;
      place(e, FaceTile<0>::CP, line, pos);
      const int g = f0 - 2 + pos;
      if (pos < TF + 3 && g >= 0 && g < nax && l0 + line < G.n[ob]) {
        const int gx0 = isx ? g : l0 + line, gy0 = isx ? l0 + line : (ax == 1 ? g : third), gz0 = ax == 2 ? g : third;
        const int64_t c = gx0 + (int64_t)G.n[0] * (gy0 + (int64_t)G.n[1] * gz0);
        if (!ECG_IN_BOUNDS(P.stats, c, nn)) continue;
#pragma unroll
        for (int f = 0; f < FL::NQ; f++) sq[f * RS + e] = P.q[(int64_t)f * nn + c];
        if (KS::NA0) sa0[e] = P.sn[(int64_t)FL::A * nn + c];
      }
    }
  }
  if (done) return;  // tested here: the staging does not wait for it
  __syncthreads();
  const double* dcc = G.dcc[ax];
  // ---- limited slopes (MUSCL, one limiter): cell f0 - 1 + s of every line, s in [0, TF]
  bool pone = true;  // no pressure read by this block's faces is below a phase's floor
  if (LSL) {
    double pf = M.eos[0].pfloor;
#pragma unroll
    for (int k = 1; k < NP; k++) pf = dmax(pf, M.eos[k].pfloor);
    const double* rdcc = G.rdcc[ax];
    for (int e = tid; e < nsl; e += FACE_THREADS) {
      int line, s;
      place(e, FaceTile<0>::LP, line, s);
      const int c = f0 - 1 + s;
      if (c < 0 || c >= nax || l0 + line >= G.n[ob]) continue;
      const int rc = line * CL + (s + 1) * PS;
      if (c == 0 || c == nax - 1) {
        // no face beyond: the missing slope is zero, and so is every limited one, except the velocity
        // along the axis at a symmetry side, whose slope there is u over the centre-to-face coordinate
        // (BoundCondWallO2Cartesian::computeSlopes :84-108)
#pragma unroll
        for (int f = 0; f < FL::NSL; f++) ssl[f * SS + e] = 0.;
        const int sd = c == 0 ? 0 : 1;
        const double wd = G.wslope[2 * ax + sd];
        if (G.bc[2 * ax + sd] == ECG_BC_SYMMETRY && fabs(wd) > 1.e-8) {
          const double* su = sq + (FL::U + ax) * RS;
          const double so = sd ? ndiv(su[rc] - su[rc - PS], dcc[c - 1]) : ndiv(su[rc + PS] - su[rc], dcc[c]);
          ssl[(3 * NP + ax) * SS + e] = limiter(code_limiter(TYPES), ndiv(su[rc], wd), so);
        }
        pone = pone && sq[FL::P * RS + rc] >= pf;
        continue;
      }
      const bool one = sq[FL::P * RS + rc - PS] >= pf && sq[FL::P * RS + rc] >= pf && sq[FL::P * RS + rc + PS] >= pf;
      pone = pone && one;
      cell_slopes<NP, DIM, code_limiter(TYPES)>(M, sq, RS, rc - PS, rc, rc + PS, dcc[c - 1], rdcc[c - 1], dcc[c], rdcc[c],
                                                one, ssl, SS, e);
    }
    pone = __syncthreads_and(pone);
  }
  // ---- face slopes (MUSCL): slope s at face g = f0 - 1 + s, between cells g-1 and g
  if (O2 && !LSL) {
    for (int e = tid; e < nsl; e += FACE_THREADS) {
      int line, s;
      place(e, FaceTile<0>::SP, line, s);
      const int gl = f0 - 2 + s;  // left cell of the face
      if (l0 + line >= G.n[ob]) continue;
      const int rl = line * CL + s * PS, rr = rl + PS;
      if (gl < 0 || gl + 1 >= nax) {
        // a side of the domain: slopes only on a symmetry side, the velocity along the axis over the
        // centre-to-face coordinate (BoundCondWallO2Cartesian::computeSlopes :84-108)
        const int sd = (gl == -1) ? 0 : ((gl == nax - 1) ? 1 : -1);
        if (sd < 0 || G.bc[2 * ax + sd] != ECG_BC_SYMMETRY) continue;
#pragma unroll
        for (int f = 0; f < FL::NSL; f++) ssl[f * SS + e] = 0.;
        const double wd = G.wslope[2 * ax + sd];
        if (fabs(wd) > 1.e-8) ssl[(3 * NP + ax) * SS + e] = ndiv(sq[(FL::U + ax) * RS + (sd ? rl : rr)], wd);
        continue;
      }
      const double d = dcc[gl];
#pragma unroll
      for (int k = 0; k < NP; k++) {
        ssl[k * SS + e] = ndiv(sq[(FL::A + k) * RS + rr] - sq[(FL::A + k) * RS + rl], d);
        ssl[(NP + k) * SS + e] = ndiv(sq[(FL::R + k) * RS + rr] - sq[(FL::R + k) * RS + rl], d);
        double pr = eos_fix_p(M.eos[k], sq[FL::P * RS + rr]), pl = eos_fix_p(M.eos[k], sq[FL::P * RS + rl]);
        ssl[(2 * NP + k) * SS + e] = ndiv(pr - pl, d);
      }
#pragma unroll
      for (int dd = 0; dd < DIM; dd++)
        ssl[(3 * NP + dd) * SS + e] = ndiv(sq[(FL::U + dd) * RS + rr] - sq[(FL::U + dd) * RS + rl], d);
    }
    __syncthreads();
  }

  // ---- one face per thread
  double wmax = wave_none(G.stretched);
  {
    int line, fl;
    place(tid, FaceTile<0>::TF, line, fl);
    const int f = f0 + fl;
    const int lg = l0 + line;
    const int rl = line * CL + (fl + 1) * PS, rr = rl + PS;  // the cells on its two sides
    const int el = line * SL + fl * PS;                      // limited slopes of the left one; face slope below
    // (bounds-checked builds: the staged cells this face reads)
    if (f <= nax && lg < G.n[ob] && ECG_IN_BOUNDS(P.stats, rl - PS, RS) && ECG_IN_BOUNDS(P.stats, rr + PS, RS)) {
      FaceAt at{f, lg, third, rl, el, pone};
      bool solved = false;
      const bool inner = f > 0 && f < nax;
      if (inner || G.bc[2 * AX + (f == 0 ? 0 : 1)] == ECG_BC_NONREFLECTING) {
        Thermo<NP> tl, tr;
        double ul[3], ur[3], Fn[3];
        Flux<NP> F;
        bool ok = true;
        if (inner) {
          face_sides<NP, DIM, AX, PASS, TYPES, false>(P, G, M, sq, at, tl, ul, tr, ur);
        } else {  // a non-reflecting side: HLLC(cell, cell) in the side's frame, with the other faces of the warp
          double ug[3];
          cell_thermo<NP, DIM, false>(M, sq, RS, f == 0 ? rr : rl, tl, ug);
          face_frame<AX>(ug, f == 0, ul);
          tr = tl;
#pragma unroll
          for (int i = 0; i < 3; i++) ur[i] = ul[i];
#pragma unroll
          for (int k = 0; k < NP; k++) ok = ok && tl.r[k] >= 1.e-15;
        }
        const double lL = G.stretched ? face_lcfl<AX>(G, f > 0 ? f - 1 : 0, lg, third) : G.lcfl;
        const double lR = G.stretched ? face_lcfl<AX>(G, f < nax ? f : nax - 1, lg, third) : G.lcfl;
        solved = hllc_quick<NP, !O2>(M, tl, ul, tr, ur, G.stretched, lL, lR, wmax, Fn, F, ok);
        if (f == 0) Fn[0] = -Fn[0];
        if (solved) store_face<NP, DIM, AX>(P, G, L.flux, f, lg, third, Fn, F);
      }
      // a symmetry side, or operands out of hllc_quick's range
      if (!solved) wmax = dmax(wmax, face_general<NP, DIM, AX, PASS, TYPES>(P, G, M0, L.flux, sq, at));
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

template <int NP, int DIM>
__device__ __forceinline__ void load_face_flux(const double* __restrict__ fl, int64_t nfa, int64_t fid, Flux<NP>& F,
                                               DevStats* st) {
  if (!ECG_IN_BOUNDS(st, fid, nfa)) fid = 0;
  const double* p = fl + fid;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    F.a[k] = p[(int64_t)k * nfa];
    F.m[k] = p[(int64_t)(NP + k) * nfa];
    F.en[k] = p[(int64_t)(2 * NP + k) * nfa];
  }
#pragma unroll
  for (int d = 0; d < DIM; d++) F.mom[d] = p[(int64_t)(3 * NP + d) * nfa];
  F.E = p[(int64_t)(3 * NP + DIM) * nfa];
  F.sM = p[(int64_t)(3 * NP + DIM + 1) * nfa];
  F.uStar = p[(int64_t)(3 * NP + DIM + 2) * nfa];
}

// How the cell kernel's loads overlap.  Accumulating face after face, a warp met the DRAM latency four (2D) to
// seven times (long-scoreboard stalls were 4.9 of 10.5 cycles between issues in 2D, DRAM at 37 %).  2D: each
// thread copies what it needs last, the Y faces' fluxes and the time-n u and E, into shared memory before its
// first load (cp.async: no registers held, 25 doubles a thread, five blocks of 128 per SM).  3D: such copies of one
// axis take 35 KB a block from L1, so a lane per component prefetches the rows of the upper faces into L2 instead
// (the lower faces' were read by earlier blocks, or are in the same rows along x).  Measured on one B200, cell
// kernels of predictor and corrector: 2D 2048^2 0.421 / 0.437 ms with neither, 0.369 / 0.381 with prefetches of the
// Y rows and the other steps, 0.323 / 0.333 with the copies; 3D 256^3 2.43 ms with neither, 2.31 / 2.33 with
// prefetches and the other steps, 2.39 / 2.47 with copies.  Prefetching for the block one wave ahead cost 30 % in 3D.
template <int NP, int DIM>
__device__ __forceinline__ void prefetch_face_fluxes(const Geometry& G, const double* const fa[3], const int g[3]) {
  using FL = Fields<NP, DIM>;
  const int c = threadIdx.x & 15;  // component; lanes 16..31 of a warp take the second 128 bytes of a row
  static_assert(FL::NFL <= 16, "a lane per component and half row");
#pragma unroll
  for (int ax = 0; ax < DIM; ax++) {
    const int64_t fid = split_fid(G.n, ax, g[ax] + 1, g[0], g[1], g[2]) - c;
    if (c < FL::NFL) asm volatile("prefetch.global.L2 [%0];" ::"l"(fa[ax] + fid + (int64_t)c * split_nfaces(G.n, ax)));
  }
}

template <int NP, int DIM, int PASS, bool PTMU, bool SEED, int TYPES>
__global__ void __launch_bounds__(cell_threads(PTMU),
                                  PTMU ? ECG_CELL_PTMU_MINB : (SEED ? ECG_CELL_SEED_MINB : ECG_CELL_MINB))
    k_kapila_cells(StepParams P, Geometry G, Model<NP> M0, const double* __restrict__ fx,
                   const double* __restrict__ fy, const double* __restrict__ fz) {
  const Model<NP> M = specialize_eos<NP, TYPES>(M0);
  using FL = Fields<NP, DIM>;
  const int done = *P.done;
  const int64_t nn = P.n;
  const int64_t cell = (int64_t)blockIdx.x * cell_threads(PTMU) + threadIdx.x;
  const bool active = cell < nn;
  int g[3] = {0, 0, 0};
  if (active) {
    g[0] = (int)(cell % G.n[0]);
    g[1] = (int)((cell / G.n[0]) % G.n[1]);
    g[2] = (int)(cell / ((int64_t)G.n[0] * G.n[1]));
  }
  double an[NP], rn[NP], pn[NP];
  double aa[NP], am[NP], ae[NP], amom[DIM], aE = 0.;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    an[k] = rn[k] = pn[k] = 0.;
    aa[k] = am[k] = ae[k] = 0.;
  }
#pragma unroll
  for (int d = 0; d < DIM; d++) amom[d] = 0.;
  CellCounters cc;
  CellPrim<NP, DIM> cp;
  const double* fa[3] = {fx, fy, fz};
  // 2D: the fluxes of the last axis' two faces, u and E of the time-n state, copied ahead into a shared slot of
  // the thread's own (no barrier)
  constexpr bool AHEAD = DIM == 2;
  constexpr int CT = cell_threads(PTMU), LA = DIM - 1;
  __shared__ double stage[AHEAD ? 2 * FL::NFL + DIM + 1 : 1][CT];
  if (active) {
    if (AHEAD) {
      const int64_t nfa = split_nfaces(G.n, LA);
      const double* lo = fa[LA] + split_fid(G.n, LA, g[LA], g[0], g[1], g[2]);
      const double* hi = fa[LA] + split_fid(G.n, LA, g[LA] + 1, g[0], g[1], g[2]);
#pragma unroll
      for (int i = 0; i < (AHEAD ? FL::NFL : 0); i++) {
        cell_copy(&stage[i][threadIdx.x], lo + (int64_t)i * nfa);
        cell_copy(&stage[FL::NFL + i][threadIdx.x], hi + (int64_t)i * nfa);
      }
#pragma unroll
      for (int d = 0; d < (AHEAD ? DIM + 1 : 0); d++)
        cell_copy(&stage[2 * FL::NFL + d][threadIdx.x], P.sn + (int64_t)(FL::U + d) * nn + cell);
    } else {
      prefetch_face_fluxes<NP, DIM>(G, fa, g);
    }
    const double p0 = P.sn[(int64_t)FL::P * nn + cell];
#pragma unroll
    for (int k = 0; k < NP; k++) {
      an[k] = P.sn[(int64_t)(FL::A + k) * nn + cell];
      rn[k] = P.sn[(int64_t)(FL::R + k) * nn + cell];
      pn[k] = eos_fix_p(M.eos[k], p0);
    }
  }
  if (done) {  // tested here: the first loads do not wait for it
    if (AHEAD) cell_copies_wait();
    return;
  }
  if (active) {
    // internal faces, axis by axis: the left face added, the right face subtracted
#pragma unroll
    for (int ax = 0; ax < DIM; ax++) {
      const int64_t nfa = split_nfaces(G.n, ax);
      const double cA = cell_coefA(G, ax, g[0], g[1], g[2]);
      Flux<NP> F;
      const bool ahead = AHEAD && ax == LA;
      if (ahead) cell_copies_wait();
      if (g[ax] >= 1) {
        if (ahead) load_face_flux<NP, DIM>(&stage[0][threadIdx.x], CT, 0, F, P.stats);
        else load_face_flux<NP, DIM>(fa[ax], nfa, split_fid(G.n, ax, g[ax], g[0], g[1], g[2]), F, P.stats);
        acc_face<NP, DIM>(cA, true, F, an, pn, aa, am, ae, amom, aE);
      }
      if (g[ax] + 1 <= G.n[ax] - 1) {
        if (ahead) load_face_flux<NP, DIM>(&stage[AHEAD ? FL::NFL : 0][threadIdx.x], CT, 0, F, P.stats);
        else load_face_flux<NP, DIM>(fa[ax], nfa, split_fid(G.n, ax, g[ax] + 1, g[0], g[1], g[2]), F, P.stats);
        acc_face<NP, DIM>(cA, false, F, an, pn, aa, am, ae, amom, aE);
      }
    }
    // the domain sides Xm, Xp, Ym, Yp, Zm, Zp, subtracted from the cell (BoundCond::computeFlux
    // src/BoundConds/BoundCond.cpp:61)
#pragma unroll
    for (int bf = 0; bf < 2 * DIM; bf++) {
      const int ax = bf >> 1;
      const bool neg = (bf & 1) == 0;
      if (neg ? (g[ax] != 0) : (g[ax] != G.n[ax] - 1)) continue;
      Flux<NP> F;
      load_face_flux<NP, DIM>(fa[ax], split_nfaces(G.n, ax), split_fid(G.n, ax, neg ? 0 : G.n[ax], g[0], g[1], g[2]),
                              F, P.stats);
      acc_face<NP, DIM>(cell_coefA(G, ax, g[0], g[1], g[2]), false, F, an, pn, aa, am, ae, amom, aE);
    }
    kapila_rebuild<NP, DIM, PASS>(P, M, nn, cell, *P.dt, an, rn, pn, aa, am, ae, amom, aE, cp,
                                  AHEAD ? &stage[AHEAD ? 2 * FL::NFL : 0][threadIdx.x] : nullptr, CT);
  }
  SeedGate<NP> sg;
  if (SEED && !PTMU) seed_gate<NP, DIM>(P, M, active, cp, sg);
  if (SEED && PTMU) ptmu_seed_gate<NP, DIM>(P, M, active, cp, sg, cc);
  if (active) kapila_finish<NP, DIM, PASS, PTMU, SEED, (TYPES == EOS_DYNAMIC)>(P, M, nn, cell, cp, sg, cc);
  block_counters<cell_threads(PTMU)>(P.stats, cc.relax, cc.iters, cc.fallback, cc.seeded, cc.rejected, cc.nonfinite, cc.ptmu, cc.iters, true);
  if (PTMU)
    block_ptmu_counters(P.stats, cc.pc.solve, cc.pc.outer, cc.pc.tsat_calls, cc.pc.tsat_iters, cc.pc.tsat_max,
                        cc.pc.seeded, cc.pc.rejected);
}

template <int NP, int DIM, int AX, int PASS, int TYPES>
cudaError_t launch_faces(const StepParams& P, const Geometry& G, const Model<NP>& M, cudaStream_t s, bool prepare) {
  using KS = FaceKernelShape<NP, DIM, PASS, TYPES>;
  auto kern = k_kapila_faces<NP, DIM, AX, PASS, TYPES>;
  const size_t sm = KS::smem_bytes();
  if (prepare) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  const FaceLaunch L = face_launch<AX>(P, KS::NA0 != 0);
  kern<<<face_grid<AX>(G.n), FACE_THREADS, sm, s>>>(P, G, M, L);
  return cudaGetLastError();
}

// One pass in split form: the face kernels of every axis, then the cell kernel.  With prepare, only
// the kernels' attributes are set.
template <int NP, int DIM, int PASS, bool PTMU, bool SEED, int TYPES>
cudaError_t launch_split(const StepParams& P, const Geometry& G, const ecg_eos* eos, double eps, cudaStream_t s,
                         bool prepare) {
  Model<NP> M;
  for (int k = 0; k < NP; k++) M.eos[k] = make_eos_params(eos[k]);
  M.eps = eps;
  const cudaError_t e = face_axes<DIM>(P, s, prepare, [&](auto ax, cudaStream_t sa) {
    return launch_faces<NP, DIM, decltype(ax)::value, PASS, TYPES>(P, G, M, sa, prepare);
  });
  if (e != cudaSuccess || prepare) return e;
  const cudaError_t ee = end_begin(P, s);
  if (ee != cudaSuccess) return ee;
  constexpr int CT = cell_threads(PTMU);
  const unsigned blocks = (unsigned)((P.n + CT - 1) / CT);
  k_kapila_cells<NP, DIM, PASS, PTMU, SEED, TYPES><<<blocks, CT, 0, s>>>(P, G, M, P.flux[0], P.flux[1],
                                                                                 DIM > 2 ? P.flux[2] : nullptr);
  const cudaError_t ec = cudaGetLastError();
  return ec == cudaSuccess ? end_join(P, s) : ec;
}

}  // namespace ecg
