// Host side of the fused whole-network kernel (ntg_chain_kernel.cuh): checks, scratch and the
// choice of an instance.
#include <string>

#include "ntg_chain_kernel.cuh"

namespace ntg {

size_t chain_smem_bytes(const ntg_chain_t& pg) {
  size_t f = 3 * (size_t)pg.channels * S0 * S0;
  for (int sgi = 0; sgi < pg.nseg; ++sgi) {
    size_t S = S0 >> sgi;
    f += 3 * S * S * pg.nconv[sgi];
  }
  return (f + 2 * NT / 32) * sizeof(float);
}

namespace {

int check_program(const std::string& w, const ntg_chain_t& pg, int& nl) {
  NTG_REQUIRE(pg.s0 == 32, w + ": the fused chain needs 32x32 inputs");
  NTG_REQUIRE(pg.nseg >= 1 && pg.nseg <= 3, w + ": 1 to 3 segments");
  NTG_REQUIRE(pg.channels >= 1 && pg.channels <= 4, w + ": 1 to 4 input channels");
  NTG_REQUIRE(pg.nconv[0] >= 1 && pg.nconv[0] <= 3, w + ": 1 to 3 convs in segment 0");
  nl = 0;
  for (int sg = 0; sg < pg.nseg; ++sg) {
    NTG_REQUIRE(pg.nconv[sg] >= 0 && pg.nconv[sg] <= 3, w + ": 0 to 3 convs per segment");
    nl += pg.nconv[sg];
  }
  NTG_REQUIRE(nl <= NTG_CHAIN_MAX_LAYERS, w + ": too many layers");
  for (int l = 0; l < nl; ++l)
    NTG_REQUIRE(pg.act[l].kind >= NTG_ACT_NONE && pg.act[l].kind <= NTG_ACT_GELU,
                w + ": unknown activation kind");
  NTG_REQUIRE(pg.readout == 0 || pg.readout == 1, w + ": readout must be 0 or 1");
  return NTG_OK;
}

// relu_only: what the networks of the Myrtle papers have in every layer, an ABRelu and the
// NTK parameterisation; rare: some layer needs the instances with every rule compiled in.
void rules_of(const ntg_chain_t& pg, int nl, bool& relu_only, bool& rare) {
  relu_only = true;
  rare = false;
  for (int l = 0; l < nl; ++l) {
    const ntg_affine_t& f = pg.aff[l];
    relu_only = relu_only && pg.act[l].kind == NTG_ACT_ABRELU && pg.act[l].stabilize <= 0.f &&
                f.nn_scaled && f.ntk_nn == 1.f && f.ntk_c == 0.f;
    rare = rare || pg.act[l].kind >= NTG_ACT_SIN;
  }
}

// Adds the parts of every pair in order.
__global__ void chain_reduce_kernel(const __grid_constant__ ntg_chain_t pg, const ChainGrid grid,
                                    const float* __restrict__ sums, int parts,
                                    float* __restrict__ out_q, float* __restrict__ out_t) {
  const int64_t pair = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pair >= grid.total) return;
  float sq = 0.f, st = 0.f;
  for (int i = 0; i < parts; ++i) {
    sq += sums[2 * (pair * parts + i)];
    st += sums[2 * (pair * parts + i) + 1];
  }
  int64_t gi, gj, o1, o2;
  chain_place(grid, pair, gi, gj, o1, o2);
  chain_write(pg, sq, st, out_q, out_t, o1, o2);
}

// The lines of the last segment in `n` runs, the longest run as short as can be: a run's cost
// is that of the segment-0 lines it takes, 32 - |d| planes and a few steps each, and the runs
// overlap by what a pooled line takes of its neighbours (six lines with three segments).
void split_lines(const ntg_chain_t& pg, int n, ChainParts& parts) {
  const int last = (S0 >> (pg.nseg - 1)) - 1;
  auto cost = [&](int a, int b) {
    int f = a, l = b;
    for (int sg = pg.nseg - 1; sg > 0; --sg) {
      const int lim = (S0 >> (sg - 1)) - 1;
      f = 2 * f - 1 < -lim ? -lim : 2 * f - 1;
      l = 2 * l + 1 > lim ? lim : 2 * l + 1;
    }
    int c = 0;
    for (int d = f; d <= l; ++d) c += S0 - (d < 0 ? -d : d) + 4;
    return c;
  };
  // the smallest bound that n greedy runs keep
  int bound = 0;
  for (int m = -last; m <= last; ++m) bound = cost(m, m) > bound ? cost(m, m) : bound;
  for (;; bound += 8) {
    int k = 0, m = -last;
    while (m <= last && k < n) {
      int e = m;
      while (e < last && cost(m, e + 1) <= bound) ++e;
      parts.first[k] = m;
      parts.last[k++] = e;
      m = e + 1;
    }
    parts.n = k;
    if (m > last) return;
  }
}

constexpr int64_t kSumFloats = 2 * kChainCtas;

int launch_chain(const char* who, const ntg_chain_t* prog, ChainArgs a, void* workspace,
                 size_t workspace_bytes) {
  const std::string w(who);
  ChainGrid& g = a.grid;
  NTG_REQUIRE(prog && a.x1 && a.x2 && a.var1 && a.var2 && a.out_q, w + ": null pointer");
  const ntg_chain_t& pg = *prog;
  int nl;
  const int rc = check_program(w, pg, nl);
  if (rc != NTG_OK) return rc;
  NTG_REQUIRE(g.n1 > 0 && g.n2 > 0 && g.r0 >= 0 && g.c0 >= 0, w + ": bad tile");
  NTG_REQUIRE(g.sym == 3 || (g.sym ? g.ld_out >= (g.r0 + g.n1 > g.c0 + g.n2 ? g.r0 + g.n1
                                                                            : g.c0 + g.n2)
                                   : g.ld_out >= g.n2),
              w + ": ld_out smaller than the kernel");
  NTG_REQUIRE(g.n1 <= (1ll << 24) && g.n2 <= (1ll << 24), w + ": tile too large");
  g.total = g.sym == 3 ? g.n1 : g.sym == 1 ? g.n1 * (g.n1 + 1) / 2 : g.n1 * g.n2;
  NTG_REQUIRE(g.total < (1ll << 31), w + ": too many pairs for one launch");
  NTG_REQUIRE(chain_smem_bytes(pg) <= 232448, w + ": network needs more shared memory than a CTA has");
  // Fewer pairs than SMs: as many parts per pair as give every SM at most one. A part repeats
  // the lines it shares with its neighbours, so beyond that a second CTA on the SM would cost
  // the first more than the shorter parts save. 35 pairs of Myrtle-5: 270 us in four parts,
  // 700 us in one.
  const int64_t fit = 152 / g.total;
  a.parts.n = 1;
  a.parts.first[0] = -((S0 >> (pg.nseg - 1)) - 1);
  a.parts.last[0] = -a.parts.first[0];
  if (fit > 1) split_lines(pg, (int)(fit < kMaxParts ? fit : kMaxParts), a.parts);
  const int64_t items = g.total * a.parts.n;
  a.ctas = items < kChainCtas ? items : kChainCtas;
  // the pooled lines' slots and the parts' sums: the caller's workspace, or stream-ordered
  // memory of our own
  const size_t need = (size_t)(a.ctas * kSlotFloats + kSumFloats) * sizeof(float);
  void* own = nullptr;
  if (workspace) {
    NTG_REQUIRE(workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0,
                w + ": workspace too small or not 16-byte aligned");
    a.slots = static_cast<float*>(workspace);
  } else {
    const cudaError_t me = cudaMallocAsync(&own, need, a.stream);
    if (me != cudaSuccess) return fail(NTG_ERR_CUDA, w + ": " + cudaGetErrorString(me));
    a.slots = static_cast<float*>(own);
  }
  a.parts.sums = a.slots + a.ctas * kSlotFloats;
  const int n0 = pg.nconv[0];
  const int c1 = pg.nseg > 1 ? pg.nconv[1] : -1, c2 = pg.nseg > 2 ? pg.nconv[2] : -1;
  cudaError_t e;
  // the Myrtle-5 / -7 / -10 shapes get kernels specialised to their segments and rules
  bool relu_only, rare;
  rules_of(pg, nl, relu_only, rare);
  if (rare)
    e = launch_chain_rare(pg, a);
  else if (pg.nseg == 3 && n0 == 2 && c1 == 1 && c2 == 1)
    e = launch_chain_myrtle5(relu_only, pg, a);
  else if (pg.nseg == 3 && n0 == 2 && c1 == 2 && c2 == 2)
    e = launch_chain_myrtle7(relu_only, pg, a);
  else if (pg.nseg == 3 && n0 == 3 && c1 == 3 && c2 == 3)
    e = launch_chain_myrtle10(relu_only, pg, a);
  else
    e = relu_only ? launch_chain_relu(pg, a) : launch_chain_any(pg, a);
  note_launch();
  if (e == cudaSuccess && a.parts.n > 1) {
    chain_reduce_kernel<<<(unsigned)ceil_div(g.total, 64), 64, 0, a.stream>>>(
        pg, g, a.parts.sums, a.parts.n, a.out_q, a.out_t);
    note_launch();
  }
  if (own) {
    const cudaError_t fe = cudaFreeAsync(own, a.stream);
    if (e == cudaSuccess) e = fe;
  }
  if (e != cudaSuccess) return fail(NTG_ERR_CUDA, w + ": " + cudaGetErrorString(e));
  return check_launch(who);
}

int sym_mode(int64_t r0, int64_t n1, int64_t c0, int64_t n2) {
  if (r0 == c0 && n1 == n2) return 1;
  return r0 + n1 <= c0 || c0 + n2 <= r0 ? 2 : -1;
}

}  // namespace
}  // namespace ntg

using namespace ntg;

extern "C" size_t ntg_chain_workspace_bytes(void) {
  return (size_t)(kChainCtas * kSlotFloats + kSumFloats) * sizeof(float);
}

extern "C" int ntg_chain_vars(void* stream, const ntg_chain_t* prog, const float* x1, int64_t n1,
                              float* var1, const float* x2, int64_t n2, float* var2,
                              void* workspace, size_t workspace_bytes) {
  const std::string w("ntg_chain_vars");
  NTG_REQUIRE(prog && x1 && var1 && workspace, w + ": null pointer");
  NTG_REQUIRE(n1 > 0 && n2 >= 0 && n1 + n2 < (1ll << 31), w + ": bad sizes");
  NTG_REQUIRE(n2 == 0 || (x2 && var2), w + ": null pointer");
  int nl;
  const int rc = check_program(w, *prog, nl);
  if (rc != NTG_OK) return rc;
  NTG_REQUIRE(workspace_bytes >= ntg_chain_workspace_bytes() &&
                  (reinterpret_cast<uintptr_t>(workspace) & 15) == 0,
              w + ": workspace too small or not 16-byte aligned");
  bool relu_only, rare;
  rules_of(*prog, nl, relu_only, rare);
  const VarArgs a{as_stream(stream), x1, n1, var1, x2, n2, var2, static_cast<float*>(workspace)};
  const cudaError_t e = rare ? launch_var_rare(*prog, a)
                        : relu_only ? launch_var_relu(*prog, a) : launch_var_any(*prog, a);
  if (e != cudaSuccess) return fail(NTG_ERR_CUDA, w + ": " + cudaGetErrorString(e));
  note_launch();
  return check_launch("ntg_chain_vars");
}

extern "C" int ntg_chain_fwd_ws(void* stream, const ntg_chain_t* prog, const float* x1,
                                const float* x2, int64_t r0, int64_t n1, int64_t c0, int64_t n2,
                                const float* var1, const float* var2, float* out_q, float* out_t,
                                int64_t ld_out, int32_t mode, void* workspace,
                                size_t workspace_bytes) {
  NTG_REQUIRE(workspace, "ntg_chain_fwd_ws: null workspace");
  ChainArgs a{as_stream(stream), x1, x2, {r0, n1, c0, n2, ld_out, 0, 0}, var1, var2, out_q,
              out_t, nullptr, 0, {}};
  if (mode == 1) {
    a.grid.sym = sym_mode(r0, n1, c0, n2);
    NTG_REQUIRE(a.grid.sym > 0 && x1 == x2,
                "ntg_chain_fwd_ws: the row and column ranges must be equal or disjoint");
  } else if (mode == 2) {
    NTG_REQUIRE(x1 == x2, "ntg_chain_fwd_ws: self pairs are of one input");
    a.grid.sym = 3;
    a.grid.n2 = 1;
  } else {
    NTG_REQUIRE(mode == 0, "ntg_chain_fwd_ws: mode must be 0, 1 or 2");
  }
  return launch_chain("ntg_chain_fwd_ws", prog, a, workspace, workspace_bytes);
}

extern "C" int ntg_chain_fwd(void* stream, const ntg_chain_t* prog, const float* x1,
                             const float* x2, int64_t r0, int64_t n1, int64_t c0, int64_t n2,
                             const float* var1, const float* var2, float* out_q, float* out_t,
                             int64_t ld_out) {
  const ChainArgs a{as_stream(stream), x1, x2, {r0, n1, c0, n2, ld_out, 0, 0}, var1, var2, out_q,
                    out_t, nullptr, 0, {}};
  return launch_chain("ntg_chain_fwd", prog, a, nullptr, 0);
}

extern "C" int ntg_chain_fwd_sym(void* stream, const ntg_chain_t* prog, const float* x,
                                 int64_t r0, int64_t n1, int64_t c0, int64_t n2, const float* var,
                                 float* out_q, float* out_t, int64_t ld_out) {
  const int sym = sym_mode(r0, n1, c0, n2);
  if (sym < 0)
    return fail(NTG_ERR_INVALID_ARG,
                "ntg_chain_fwd_sym: the row and column ranges must be equal or disjoint");
  const ChainArgs a{as_stream(stream), x, x, {r0, n1, c0, n2, ld_out, sym, 0}, var, var, out_q,
                    out_t, nullptr, 0, {}};
  return launch_chain("ntg_chain_fwd_sym", prog, a, nullptr, 0);
}
