// Instances of the fused chain's variance kernel.
#include "ntg_chain_kernel.cuh"

namespace ntg {
namespace {

template <int RO, int KC = 0>
cudaError_t by_convs(const ntg_chain_t& pg, const VarArgs& a) {
  switch (pg.nconv[0]) {
    case 1: return launch_var_k<1, RO, KC>(pg, a);
    case 2: return launch_var_k<2, RO, KC>(pg, a);
    default: return launch_var_k<3, RO, KC>(pg, a);
  }
}

}  // namespace

cudaError_t launch_var_relu(const ntg_chain_t& pg, const VarArgs& a) {
  return pg.channels == 3 ? by_convs<1, 3>(pg, a) : by_convs<1>(pg, a);
}
cudaError_t launch_var_any(const ntg_chain_t& pg, const VarArgs& a) { return by_convs<0>(pg, a); }
cudaError_t launch_var_rare(const ntg_chain_t& pg, const VarArgs& a) { return by_convs<2>(pg, a); }

}  // namespace ntg
