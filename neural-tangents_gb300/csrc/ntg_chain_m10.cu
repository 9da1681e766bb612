// Instances of the fused chain kernel for segments of 3, 3, 3 convs.
#include "ntg_chain_kernel.cuh"

namespace ntg {

cudaError_t launch_chain_myrtle10(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a) {
  return launch_myrtle<3, 3, 3>(relu_only, pg, a);
}

}  // namespace ntg
