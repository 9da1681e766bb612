// Instances of the fused chain kernel for any segment shape with an ABRelu in every layer
// (NTK parameterisation).
#include "ntg_chain_kernel.cuh"

namespace ntg {

cudaError_t launch_chain_relu(const ntg_chain_t& pg, const ChainArgs& a) {
  switch (pg.nconv[0]) {
    case 1: return launch_chain_k<1, 0, 0, 0, 1>(pg, a);
    case 2: return launch_chain_k<2, 0, 0, 0, 1>(pg, a);
    default: return launch_chain_k<3, 0, 0, 0, 1>(pg, a);
  }
}

}  // namespace ntg
