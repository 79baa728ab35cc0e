// Face launches of the split forms (ecg_kapila_split.cuh, ecg_flow_split.cuh): the grids of every axis' faces,
// their tiles (FaceTile, ecg_tma.cuh) and the face arrays.
#pragma once
#include <type_traits>

#include "ecg_step.cuh"
#include "ecg_tma.cuh"

namespace ecg {

// Index of a face in its axis' face array: the face between cells f-1 and f along AX (f = 0 and f = n_AX are
// the domain sides) of the line at the other coordinates, so that consecutive threads of either kernel touch
// consecutive faces.
__device__ __forceinline__ int64_t split_fid(const int n[3], int ax, int f, int i, int j, int k) {
  if (ax == 0) return (int64_t)f + (int64_t)(n[0] + 1) * ((int64_t)j + (int64_t)n[1] * k);
  if (ax == 1) return (int64_t)i + (int64_t)n[0] * ((int64_t)f + (int64_t)(n[1] + 1) * k);
  return (int64_t)i + (int64_t)n[0] * ((int64_t)j + (int64_t)n[1] * f);
}

// What a face kernel needs beside the step's parameters: its axis' face array and the tensor maps of the
// staged buffers (tma: they apply).
struct FaceLaunch {
  CUtensorMap q, a0;
  double* flux;
  int tma;
};

// Copies of a cell kernel's later inputs into shared slots of the thread's own, issued before its first load
// (cp.async: no registers held, no barrier needed).
__device__ __forceinline__ void cell_copy(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cell_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The face arrays a cell kernel reads.
struct FaceArrays {
  const double* flux[3];
};

// Grid of the faces normal to AX: chunks of TF faces along it times groups of W lines, for every third
// coordinate (Z for X and Y faces, Y for Z faces); x runs along the staged rows.
template <int AX>
inline dim3 face_grid(const int n[3]) {
  using FT = FaceTile<AX>;
  const unsigned gf = (unsigned)((n[AX] + 1 + FT::TF - 1) / FT::TF);
  const unsigned gl = (unsigned)((n[AX == 0 ? 1 : 0] + FT::W - 1) / FT::W), third = (unsigned)(AX == 2 ? n[1] : n[2]);
  return AX == 0 ? dim3(gf, gl, third) : dim3(gl, gf, third);
}
struct FacePlace {
  int f0, l0, third;
};
template <int AX>
__device__ __forceinline__ FacePlace face_place() {
  return {(int)(AX == 0 ? blockIdx.x : blockIdx.y) * FaceTile<AX>::TF, (int)(AX == 0 ? blockIdx.y : blockIdx.x) * FaceTile<AX>::W,
          (int)blockIdx.z};
}

// The launch record of axis AX: tensor maps of the buffers the pass reads, where the context built them
// (need_a0: the kernel stages the time-n alpha_0 plane too).
template <int AX>
inline FaceLaunch face_launch(const StepParams& P, bool need_a0) {
  FaceLaunch L{};
  L.flux = P.flux[AX];
  if (P.fmaps && P.fmaps->ok) {
    int q = -1, a = -1;
    for (int b = 0; b < 3; b++) {
      if (P.fmaps->buf[b] && P.fmaps->buf[b] == P.q) q = b;
      if (P.fmaps->buf[b] && P.fmaps->buf[b] == P.sn) a = b;
    }
    if (q >= 0 && (!need_a0 || a >= 0)) {
      L.q = P.fmaps->q[q][AX];
      if (a >= 0) L.a0 = P.fmaps->a0[a][AX];
      L.tma = 1;
    }
  }
  return L;
}

// Launches the face kernels of every axis side by side: X on the step's stream, the others on the context's
// auxiliary streams, forked from it and joined to it by events (branches of the graph when the step is
// captured).  They are independent, and one after another each waited for the last wave of the one before and,
// on small meshes, for its whole latency.  Measured side by side against one after another (one B200,
// mid-run states, per step): 191 x 103 cells 109 -> 95 us, 1000 x 601 with THINC 636 -> 598 us, 67 x 53 x 61
// 427 -> 408 us; 2048^2 and 256^3 unchanged.
// One kernel for all axes instead measured slower: with a copy of the code per axis 8 % (256^3) to 10 %
// (2048^2) in the face work, with the axis as run-time strides 11 %.
// Profiled steps (split_ev) run them in order, an event after each.
template <int DIM, class F>
inline cudaError_t face_axes(const StepParams& P, cudaStream_t s, bool prepare, F&& launch) {
  const FaceStreams* fs = (prepare || P.split_ev) ? nullptr : P.fstreams;
  cudaError_t e = cudaSuccess;
  if (fs) e = cudaEventRecord(fs->fork, s);
  auto one = [&](auto ax) {
    constexpr int a = decltype(ax)::value;
    if (e != cudaSuccess) return;
    cudaStream_t sa = s;
    if (fs && a > 0) {
      sa = fs->s[a - 1];
      e = cudaStreamWaitEvent(sa, fs->fork, 0);
    }
    if (e == cudaSuccess) e = launch(ax, sa);
    if (e == cudaSuccess && !prepare && P.split_ev) e = cudaEventRecord(P.split_ev[a], s);
    if (e == cudaSuccess && sa != s) e = cudaEventRecord(fs->join[a - 1], sa);
  };
  one(std::integral_constant<int, 0>{});
  one(std::integral_constant<int, 1>{});
  if constexpr (DIM > 2) one(std::integral_constant<int, 2>{});
  for (int a = 1; fs && a < DIM && e == cudaSuccess; a++) e = cudaStreamWaitEvent(s, fs->join[a - 1], 0);
  return e;
}

// The end of the step beside its last cell kernel: the wave speeds are complete once the face kernels are, and
// the cell kernel reads the scalars of its own parity.
cudaError_t launch_step_end(const DevScalars* from, DevScalars* to, cudaStream_t s);
inline cudaError_t end_begin(const StepParams& P, cudaStream_t s) {
  if (!P.end) return cudaSuccess;
  cudaError_t e = cudaEventRecord(P.end->fork, s);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(P.end->s, P.end->fork, 0);
  if (e == cudaSuccess) e = launch_step_end(P.end->from, P.end->to, P.end->s);
  if (e == cudaSuccess) e = cudaEventRecord(P.end->join, P.end->s);
  return e;
}
inline cudaError_t end_join(const StepParams& P, cudaStream_t s) {
  return P.end ? cudaStreamWaitEvent(s, P.end->join, 0) : cudaSuccess;
}

}  // namespace ecg
