// Euler step passes in split form on 2D meshes.
#include "ecg_euler.cuh"

namespace ecg {

cudaError_t euler_flow_2d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, double eps,
                          cudaStream_t s, bool prepare) {
  return euler_flow<2>(pass, P, G, eos, eps, s, prepare);
}

}  // namespace ecg
