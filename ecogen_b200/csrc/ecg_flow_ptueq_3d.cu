// PTUEq step passes in split form on 3D meshes.
#include "ecg_ptueq.cuh"

namespace ecg {

cudaError_t ptueq_flow_3d(int pass, const StepParams& P, const Geometry& G, const ecg_eos* eos, cudaStream_t s,
                          bool prepare) {
  return ptueq_flow<3>(pass, P, G, eos, s, prepare);
}

}  // namespace ecg
