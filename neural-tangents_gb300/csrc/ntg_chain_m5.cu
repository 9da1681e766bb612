// Instances of the fused chain kernel for segments of 2, 1, 1 convs.
#include "ntg_chain_kernel.cuh"

namespace ntg {

cudaError_t launch_chain_myrtle5(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a) {
  return launch_myrtle<2, 1, 1>(relu_only, pg, a);
}

}  // namespace ntg
