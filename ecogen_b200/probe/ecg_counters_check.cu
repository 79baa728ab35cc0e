// Check of the step kernels' per-block counter reduction (block_counters, csrc/ecg_step.cuh) for blocks of 32 to 1024
// threads: the same hashed per-thread counters added one by one on the host.  Test infrastructure, built into the
// probe library (libecg_probe.so), not part of the solver's C ABI.
#include <cuda_runtime.h>

#include <cstring>

#include "../csrc/ecg_step.cuh"

using namespace ecg;

namespace {

struct Counters {
  unsigned int relax, iters, fallback, seeded, rejected, nonfinite, ptmu, max_iters;
};

__host__ __device__ inline Counters draw(unsigned long long seed, unsigned int t) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (t + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  Counters c;
  c.relax = (unsigned int)(z & 3) != 0;
  c.iters = c.relax ? (unsigned int)((z >> 2) % 21) : 0u;
  const bool rare = ((z >> 8) & 63) == 0;  // most warps have none of these
  c.fallback = rare && ((z >> 16) & 1);
  c.seeded = rare && ((z >> 17) & 1);
  c.rejected = rare && ((z >> 18) & 1);
  c.nonfinite = rare && ((z >> 19) & 1);
  c.ptmu = rare && ((z >> 20) & 1);
  c.max_iters = c.iters;
  return c;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_counters(unsigned long long seed, DevStats* st) {
  const Counters c = draw(seed, blockIdx.x * THREADS + threadIdx.x);
  block_counters<THREADS>(st, c.relax, c.iters, c.fallback, c.seeded, c.rejected, c.nonfinite, c.ptmu, c.max_iters, true);
}

}  // namespace

// blocks blocks of `threads` (32, 64, 128, 256, 512 or 1024) threads; got and want receive the 24 counters in
// DevStats' order.  Returns 0, a CUDA error code, or -1 for arguments outside the limits.
extern "C" int ecg_probe_counters(unsigned long long seed, int blocks, int threads, unsigned long long got[24],
                                  unsigned long long want[24]) {
  if (blocks < 1 || blocks > 4096) return -1;
  DevStats* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(DevStats));
  if (e != cudaSuccess) return (int)e;
  e = cudaMemset(d, 0, sizeof(DevStats));
  if (e == cudaSuccess) {
    switch (threads) {
      case 32: k_counters<32><<<blocks, 32>>>(seed, d); break;
      case 64: k_counters<64><<<blocks, 64>>>(seed, d); break;
      case 128: k_counters<128><<<blocks, 128>>>(seed, d); break;
      case 256: k_counters<256><<<blocks, 256>>>(seed, d); break;
      case 512: k_counters<512><<<blocks, 512>>>(seed, d); break;
      case 1024: k_counters<1024><<<blocks, 1024>>>(seed, d); break;
      default: cudaFree(d); return -1;
    }
    e = cudaGetLastError();
  }
  DevStats h{};
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  std::memcpy(got, &h, 24 * sizeof(unsigned long long));
  DevStats w{};
  for (unsigned int t = 0; t < (unsigned int)(blocks * threads); t++) {
    const Counters c = draw(seed, t);
    w.relax_calls += c.relax;
    w.newton_evals += c.iters;
    w.newton_fallback += c.fallback;
    w.seeded += c.seeded;
    w.seed_rejected += c.rejected;
    w.nonfinite += c.nonfinite;
    w.ptmu_errors += c.ptmu;
    if (c.max_iters > w.newton_max) w.newton_max = c.max_iters;
    if (c.relax) w.hist[c.iters < 16 ? (c.iters >= 1 ? c.iters - 1 : 0) : 15]++;
  }
  std::memcpy(want, &w, 24 * sizeof(unsigned long long));
  return (int)e;
}
