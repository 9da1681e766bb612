// Fused whole-network NNGP/NTK kernel for the Myrtle conv-net family on sm_103a.
//
// One CTA computes one (x1[i], x2[j]) pair end to end: first-layer Gram ->
// [3x3 SAME Conv + activation] x n0 -> AvgPool(2) -> [Conv + act] x n1 ->
// AvgPool(2) -> ... -> readout (mean of all spatial entries, or the mean of the
// spatial diagonal).  Nothing but the two readout scalars reaches HBM.
//
// Data layout.  The full-spatial kernel K[h, h', w, w'] of a pair is walked
// along its "lines": a line is the set of planes (h, h + delta) for a fixed
// delta; every Conv rule only couples planes of the same line
// (K'[h,h',..] = sum_d K[h+d, h'+d, ..]).  Inside a plane the (w, w') square is
// stored skewed: row r = (w' - w) mod S, column c = w, so the w-direction
// stencil neighbours (w +- 1, w' +- 1) are column neighbours of the same row
// (a row holds two diagonals of the square, split at c = S - r).  A thread owns
// consecutive columns of one row in every plane of a line; the h-direction
// stencil is a 3-plane register ring, the w-direction one two warp shuffles.
// AvgPool(2) couples lines 2m-1, 2m, 2m+1 into pooled line m; a completed pooled
// line is processed by the next segment right away.
//
// Bound by FP32 issue and the latency of an entry's dependent chain, not by memory.
// So two CTAs of 256 threads share an SM (four columns a thread at 32 x 32: two
// independent packed chains each), one filling the other's barriers and its narrow
// later segments; what that takes in shared memory is bought by keeping the pooled
// lines (64 KB) in L2, where nothing waits for them (red.add, read one plane
// ahead), and no square roots of the variances. K(x, x) of 120 images through Myrtle-5
// (7260 pairs): 41.0 ms with one CTA of 512 threads, two columns a thread and the pooled
// lines in shared memory (4.56 M warp instructions a pair, 65 % of the issue slots), 25.1 ms
// so (2.7 M, 64 %). Three CTAs an SM (80 registers, spills): 27.1 ms; the layers of a step
// made independent of one another (each on the plane of the step before, 128 registers):
// 27.0 ms.
#pragma once

#include <type_traits>

#include "ntg_common.cuh"

namespace ntg {

constexpr int NT = 256;
constexpr int S0 = 32, S1 = 16, S2 = 8;

// A pooled line of a segment of size H: [parity][tensor][plane] of H + H / 2 rows of H floats,
// the H skewed rows and one side row per warp of the segment before (see chain_line).
template <int H>
constexpr int slot_plane() {
  return (H + H / 2) * H;
}
constexpr int kSlots1 = 4 * S1 * slot_plane<S1>();
constexpr int kSlots2 = 4 * S2 * slot_plane<S2>();
constexpr int64_t kSlotFloats = kSlots1 + kSlots2;  // one CTA's
constexpr int kChainCtasPerSm = 2;
constexpr int64_t kChainCtas = kChainCtasPerSm * 152;

// Few pairs: each is split into `n` parts, part i the lines first[i] .. last[i] of the last
// segment (and the lines of the segments before that these take), on a CTA each; the parts'
// sums go to `sums` [pair][part][2] and are added in order by chain_reduce_kernel.
constexpr int kMaxParts = 8;
struct ChainParts {
  int n;
  int first[kMaxParts], last[kMaxParts];
  float* sums;
};

// Where pair `pair` of a launch comes from and goes to (see chain_fwd_kernel).
struct ChainGrid {
  int64_t r0, n1, c0, n2, ld_out;
  int sym;
  int64_t total;
};

struct ChainArgs {
  cudaStream_t stream;
  const float *x1, *x2;
  ChainGrid grid;
  const float *var1, *var2;
  float *out_q, *out_t;
  float* slots;
  int64_t ctas;
  ChainParts parts;
};

struct VarArgs {
  cudaStream_t stream;
  const float* x1;
  int64_t n1;
  float* var1;
  const float* x2;
  int64_t n2;
  float* var2;
  float* slots;
};

// One function per group of kernel instances, each in its own translation unit (the whole
// set takes minutes in one).
cudaError_t launch_chain_myrtle5(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_chain_myrtle7(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_chain_myrtle10(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_chain_relu(const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_chain_any(const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_chain_rare(const ntg_chain_t& pg, const ChainArgs& a);
cudaError_t launch_var_relu(const ntg_chain_t& pg, const VarArgs& a);
cudaError_t launch_var_any(const ntg_chain_t& pg, const VarArgs& a);
cudaError_t launch_var_rare(const ntg_chain_t& pg, const VarArgs& a);
size_t chain_smem_bytes(const ntg_chain_t& pg);

namespace {

struct ChainCtx {
  int K;
  float inv_k;
  float acc_q, acc_t;  // per-thread readout partial sums
  int readout;
};

__device__ __forceinline__ void red_add(float* p, const float (&v)[2]) {
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v[0]), "f"(v[1])
               : "memory");
}
__device__ __forceinline__ void red_add(float* p, const float (&v)[1]) {
  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p), "f"(v[0]) : "memory");
}
__device__ __forceinline__ void put(float* p, const float (&v)[2]) {
  *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
__device__ __forceinline__ void put(float* p, const float (&v)[1]) { *p = v[0]; }

// Processes line `delta` of a segment of size S with NC conv layers: a thread owns NP packed
// f32x2 pairs of consecutive columns (four entries at S = 32, two below) of one skewed row in
// every plane of the line, eight threads a row (four at S = 8), so a warp holds whole rows,
// the w-direction stencil is two shuffles per tensor and thread, and at S = 32 two packed
// chains per thread are in flight. Threads past the plane leave at once; no barrier inside.
// FIRST: level-0 input is the first-layer Gram of the two images (its NTK is the scalar zero
// of an input kernel); otherwise it is pooled line `delta` of in_slots, scaled by 1/16 for the
// AvgPool normalisation. LAST: the final level feeds the readout sums, otherwise it is
// average-pooled into out_slots: a pooled entry (rho, j) takes columns 2j, 2j + 1 of row
// 2 rho, column 2j of row 2 rho + 1 and column 2j + 1 of row 2 rho - 1. The thread of row
// 2 rho adds them up (two shuffles) but for a warp's first row, whose row 2 rho - 1 is the
// last of the warp before: that one adds its column to a side row of its own, which the
// reader of the line adds, so warps never wait for one another. Each thread's additions to an
// entry come in the order of lines and planes (a fixed one); plane (1, 0) of the window, an
// odd plane of an odd line, comes first and stores.
// `sec`: the segment's planes in shared memory, three sections of (images when FIRST, then one
// variance map per layer) S x S planes each: sample 1, sample 2, and sample 2 shifted one
// column left ([row][j] = [row][j + 1]), so that the sample-2 entries of a pair are one
// aligned 8-byte load on odd rows too, and an address per sample serves every plane of it.
// RO: what is compiled in: 1: an ABRelu in every layer, NTK parameterisation, 0: ABRelu, Erf
// or no activation, 2: every rule (Sin / Rbf / Gelu as well). ROOTS: see abrelu2_v; always with
// RO 0 and 2. COMP: see abrelu2.
// KC > 0: channel count. NTK = false: the nngp only (the ntk's slots are left alone).
template <int S, int NC, bool FIRST, bool LAST, int RO, bool ROOTS, int COMP, int KC,
          bool NTK = true>
__device__ __forceinline__ void chain_line(ChainCtx& cx, const ntg_chain_t& pg, int lbase,
                                           const float* sec, const float* in_slots,
                                           float* out_slots, int delta) {
  constexpr int NP = S >= 16 ? S / 16 : 1;  // packed pairs per thread
  constexpr int TPR = S / (2 * NP);         // threads of a row
  constexpr int USED = TPR * S;             // whole warps
  static_assert(USED % 32 == 0 && USED <= NT, "rows must tile warps");
  static_assert(LAST || TPR == 8, "pooling shuffles assume rows 8 lanes apart");
  const int tid = threadIdx.x;
  if (USED < NT && tid >= USED) return;
  const int lane = tid & 31;
  const int r = tid / TPR, c0 = (tid % TPR) * 2 * NP;
  const int lo = delta < 0 ? -delta : 0;
  const int hi = delta < 0 ? S : S - delta;
  const int K = FIRST ? (KC > 0 ? KC : cx.K) : 0;
  const int D = (K + NC) * S * S;  // floats of a section

  // 1/0 weights of the left / right C-direction stencil neighbours (zero at the row ends and
  // at the split between the row's two diagonals)
  float ml[2 * NP], mr[2 * NP];
#pragma unroll
  for (int u = 0; u < 2 * NP; ++u) {
    const int c = c0 + u;
    ml[u] = (c >= 1 && c != S - r) ? 1.f : 0.f;
    mr[u] = (c <= S - 2 && c != S - 1 - r) ? 1.f : 0.f;
  }
  // row `s` of sample 1 at a1, row s + delta of sample 2 at a2[u]; both advance by a row
  const float* a1 = sec + lo * S + c0;
  const float* a2[NP];
#pragma unroll
  for (int u = 0; u < NP; ++u) {
    const int wp = (c0 + 2 * u + r) & (S - 1);
    a2[u] = sec + ((r & 1) ? 2 * D + wp - 1 : D + wp) + (lo + delta) * S;
  }
  const P2 zero = p2s(0.f);

  constexpr int NA = NC > 0 ? NC : 1;
  ActC acs[NA];
#pragma unroll
  for (int k = 0; k < NC; ++k) acs[k] = act_consts(pg.act[lbase + k]);
  const P2 INVK = p2s(cx.inv_k);

  // ring of the last two planes of every conv layer's input
  P2 Aq[NA][NP], Bq[NA][NP], At[NA][NP], Bt[NA][NP];
#pragma unroll
  for (int k = 0; k < NC; ++k)
#pragma unroll
    for (int u = 0; u < NP; ++u) Aq[k][u] = Bq[k][u] = At[k][u] = Bt[k][u] = zero;

  // a pooled plane is read from L2 one plane ahead: rows, and the side rows of even ones
  P2 fq[NP], ft[NP], gq[NP], gt[NP];
  constexpr int IP = slot_plane<S>();
  const float* in = nullptr;
  if (!FIRST) in = in_slots + (2 * (delta & 1)) * (S * IP) + lo * IP + c0;
  const int side = (S + ((r / 2 + S / 2 - 1) % (S / 2))) * S;
  auto fetch = [&]() {
#pragma unroll
    for (int u = 0; u < NP; ++u) {
      const float* p = in + 2 * u;
      fq[u].v = __ldcg(reinterpret_cast<const unsigned long long*>(p + r * S));
      ft[u] = gq[u] = gt[u] = zero;
      if (NTK) ft[u].v = __ldcg(reinterpret_cast<const unsigned long long*>(p + S * IP + r * S));
      if ((r & 1) == 0) {
        gq[u].v = __ldcg(reinterpret_cast<const unsigned long long*>(p + side));
        if (NTK)
          gt[u].v = __ldcg(reinterpret_cast<const unsigned long long*>(p + S * IP + side));
      }
    }
    in += IP;
  };
  if (!FIRST) fetch();

  // where this thread's pooled sums go: planes p even / odd, the line they belong to
  constexpr int H = S / 2, OP = slot_plane<H>();
  float *oe = nullptr, *oo = nullptr;
  bool adds = false;
  const float mup = lane >= 24 ? 0.f : 1.f, mdn = lane >= 24 || lane < 8 ? 0.f : 1.f;
  if (!LAST) {
    const int row = lane >= 24 ? H + (tid >> 5) : r >> 1;
    const int me = (delta & 1) ? (delta - 1) / 2 : delta / 2;
    const int mo = (delta & 1) ? me + 1 : me;
    oe = out_slots + (2 * (me & 1)) * (H * OP) + row * H + c0 / 2;
    oo = out_slots + (2 * (mo & 1)) * (H * OP) + row * H + c0 / 2;
    adds = (lane & 8) == 0 || lane >= 24;
  }

  // one plane step; FULL: every level is inside the line
  auto step = [&](int s, auto full) {
    constexpr bool FULL = decltype(full)::value;
    // ---- level 0 at plane s ----
    P2 nq[NP], nt[NP];
#pragma unroll
    for (int u = 0; u < NP; ++u) nq[u] = nt[u] = zero;
    if (FULL || s < hi) {
      if (FIRST) {
        // first-layer Gram of the two images, channel by channel in the same order as
        // ntg_input_fs, so that both paths round alike
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < K) {
#pragma unroll
            for (int u = 0; u < NP; ++u)
              nq[u] = fma2(p2ld(a1 + k * (S * S) + 2 * u), p2ld(a2[u] + k * (S * S)), nq[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < NP; ++u) nq[u] = mul2(nq[u], INVK);
      } else {
        const P2 sc = p2s(0.0625f);
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          nq[u] = mul2(add2(fq[u], gq[u]), sc);
          nt[u] = mul2(add2(ft[u], gt[u]), sc);
        }
        if (s + 1 < hi) fetch();
      }
    }
    // ---- conv layers: level k + 1 at plane s - k - 1 ----
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const int p = s - k - 1;
      const bool has_t = NTK && !(FIRST && k == 0);
      float hq[2 * NP], ht[2 * NP];
#pragma unroll
      for (int u = 0; u < NP; ++u) {
        p2u(add2(add2(Aq[k][u], Bq[k][u]), nq[u]), hq[2 * u], hq[2 * u + 1]);
        if (has_t) p2u(add2(add2(At[k][u], Bt[k][u]), nt[u]), ht[2 * u], ht[2 * u + 1]);
        Aq[k][u] = Bq[k][u];
        Bq[k][u] = nq[u];
        At[k][u] = Bt[k][u];
        Bt[k][u] = nt[u];
        if (!FULL) nq[u] = nt[u] = zero;
      }
      if (FULL || (p >= lo && p < hi)) {  // uniform across the CTA
        const ntg_affine_t& af = pg.aff[lbase + k];
        const ActC& ac = acs[k];
        // the w-direction stencil, (h + ml * left) + mr * right per entry
        const float lq = __shfl_up_sync(0xffffffffu, hq[2 * NP - 1], 1);
        const float rq = __shfl_down_sync(0xffffffffu, hq[0], 1);
        float lt = 0.f, rt = 0.f;
        if (has_t) {
          lt = __shfl_up_sync(0xffffffffu, ht[2 * NP - 1], 1);
          rt = __shfl_down_sync(0xffffffffu, ht[0], 1);
        }
        float cq[2 * NP], ct[2 * NP];
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u) {
          cq[u] = fmaf(mr[u], u + 1 < 2 * NP ? hq[u + 1] : rq,
                       fmaf(ml[u], u > 0 ? hq[u - 1] : lq, hq[u]));
          ct[u] = has_t ? fmaf(mr[u], u + 1 < 2 * NP ? ht[u + 1] : rt,
                               fmaf(ml[u], u > 0 ? ht[u - 1] : lt, ht[u]))
                        : 0.f;
        }
        const P2 W2 = p2s(af.w2 * (1.f / 9.f)), B2 = p2s(af.b2);
        const P2 TW = p2s(af.ntk_w2 * (1.f / 9.f));
        const int vo = (K + k) * S * S - (k + 1) * S;  // layer k's map at plane p
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          const P2 c2 = p2(cq[2 * u], cq[2 * u + 1]), t2 = p2(ct[2 * u], ct[2 * u + 1]);
          P2 q = fma2(W2, c2, B2), t;
          if (!NTK) {
            t = zero;
          } else if (RO == 1) {  // ntk = nngp + W^2 ntk_in
            t = has_t ? fma2(TW, t2, q) : q;
          } else {
            const P2 nn = af.nn_scaled ? q : mul2(c2, p2s(1.f / 9.f));
            t = fma2(TW, t2, fma2(p2s(af.ntk_nn), nn, p2s(af.ntk_c)));
          }
          if (RO == 1 || ac.kind != NTG_ACT_NONE) {
            const P2 v1 = p2ld(a1 + vo + 2 * u), v2 = p2ld(a2[u] + vo);
            if (RO == 1 || (ac.kind == NTG_ACT_ABRELU && ac.stab <= 0.f)) {
              abrelu2_v<COMP, ROOTS>(ac, q, t, v1, v2);
            } else {
              float qa, qb, ta, tb, va, vb, wa, wb;
              p2u(q, qa, qb);
              p2u(t, ta, tb);
              p2u(v1, va, vb);
              p2u(v2, wa, wb);
              act_apply<RO == 2>(ac, qa, ta, va, wa, sqrt_var(va), sqrt_var(wa));
              act_apply<RO == 2>(ac, qb, tb, vb, wb, sqrt_var(vb), sqrt_var(wb));
              q = p2(qa, qb);
              t = p2(ta, tb);
            }
          }
          nq[u] = q;
          nt[u] = t;
        }
      }
    }
    a1 += S;
#pragma unroll
    for (int u = 0; u < NP; ++u) a2[u] += S;
    // ---- emit the last level at plane p = s - NC ----
    const int p = s - NC;
    if (!FULL && (p < lo || p >= hi)) return;
    float q[2 * NP], t[2 * NP];
#pragma unroll
    for (int u = 0; u < NP; ++u) {
      p2u(nq[u], q[2 * u], q[2 * u + 1]);
      p2u(nt[u], t[2 * u], t[2 * u + 1]);
    }
    if (LAST) {
      if (cx.readout == 0 || (delta == 0 && r == 0)) {
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          cx.acc_q += q[2 * u] + q[2 * u + 1];
          cx.acc_t += t[2 * u] + t[2 * u + 1];
        }
      }
    } else {
      float vq[NP], vt[NP];
#pragma unroll
      for (int u = 0; u < NP; ++u) {
        const float uq = __shfl_down_sync(0xffffffffu, q[2 * u], 8);
        const float ut = NTK ? __shfl_down_sync(0xffffffffu, t[2 * u], 8) : 0.f;
        const float dq = __shfl_up_sync(0xffffffffu, q[2 * u + 1], 8);
        const float dt = NTK ? __shfl_up_sync(0xffffffffu, t[2 * u + 1], 8) : 0.f;
        // a whole window; without row 2 rho - 1 in a warp's first row; the side row's column
        vq[u] = fmaf(mup, q[2 * u] + uq, fmaf(mdn, dq, q[2 * u + 1]));
        vt[u] = fmaf(mup, t[2 * u] + ut, fmaf(mdn, dt, t[2 * u + 1]));
      }
      float* o = ((p & 1) ? oo : oe) + (p >> 1) * OP;
      if (adds) {
        if ((delta & 1) && (p & 1)) {
          put(o, vq);
          if (NTK) put(o + H * OP, vt);
        } else {
          red_add(o, vq);
          if (NTK) red_add(o + H * OP, vt);
        }
      }
    }
  };

  // planes with every level inside the line, by threes (the period of the (A, B, new) plane
  // ring, so that its rotation is a renaming of registers); the others one by one. With more than
  // the ReLU rule compiled in (RO 0 and 2, always ROOTS) four copies of a step are more code than
  // the SM's instruction cache holds: 60 images through Myrtle-5 with Erf 19.1 ms so and 14.2 one
  // by one, Gelu 45.3 and 35.2, Sin 27.4 and 18.7, Myrtle-10 with Erf 44.0 and 26.1.
  int s = lo;
  while (s < hi + NC) {
    if (S == S0 && !ROOTS && s >= lo + NC && s + 2 < hi) {
      step(s, std::true_type());
      step(s + 1, std::true_type());
      step(s + 2, std::true_type());
      s += 3;
    } else {
      step(s, std::false_type());
      ++s;
    }
  }
}

// NCT >= 0: the segment's conv count is known at compile time (one instantiation).
template <int S, bool LAST, int NCT, int RO, bool ROOTS, int COMP, bool NTK = true>
__device__ __forceinline__ void pooled_line(ChainCtx& cx, const ntg_chain_t& pg, int ncv,
                                            int lbase, const float* sec, const float* in_slots,
                                            float* out_slots, int m) {
  auto line = [&](auto nc) {
    chain_line<S, decltype(nc)::value, false, LAST, RO, ROOTS, COMP, 0, NTK>(
        cx, pg, lbase, sec, in_slots, out_slots, m);
  };
  if constexpr (NCT >= 0) {
    line(std::integral_constant<int, NCT>());
    return;
  }
  switch (ncv) {
    case 0: line(std::integral_constant<int, 0>()); break;
    case 1: line(std::integral_constant<int, 1>()); break;
    case 2: line(std::integral_constant<int, 2>()); break;
    default: line(std::integral_constant<int, 3>()); break;
  }
}

// Segment sizes 32 -> 16 -> 8 (nseg <= 3); segment 0 has N0 conv layers.
// Pair p of the upper triangle (i <= j) of an n x n grid, row by row.
__device__ __forceinline__ void tri_pair(int64_t p, int64_t n, int64_t& i, int64_t& j) {
  auto start = [&](int64_t r) { return r * n - (r * (r - 1)) / 2; };  // first pair of row r
  const double b = 2.0 * (double)n + 1.0;
  int64_t r = (int64_t)floor((b - sqrt(fmax(b * b - 8.0 * (double)p, 0.0))) * 0.5);
  if (r < 0) r = 0;
  if (r > n - 1) r = n - 1;
  while (r > 0 && start(r) > p) --r;
  while (r + 1 < n && start(r + 1) <= p) ++r;
  i = r;
  j = r + (p - start(r));
}

// One sample pair's images (as channel planes) and variance maps into the sections that
// chain_line reads, segment by segment; returns the first float after them. one_root: whether
// the variances that this thread loaded are all one_root_var.
__device__ __forceinline__ float* load_pair(ChainCtx& cx, const ntg_chain_t& pg, int nseg,
                                            const float* im1, const float* im2, const float* g1,
                                            const float* g2, float* smem, float* (&sec)[3],
                                            bool& one_root) {
  const int K = pg.channels;
  float* p = smem;
  int l = 0;
  for (int sgi = 0; sgi < nseg; ++sgi) {
    const int S = S0 >> sgi, n = S * S, nc = pg.nconv[sgi];
    const int D = ((sgi == 0 ? K : 0) + nc) * n;
    sec[sgi] = p;
    if (sgi == 0) {
      for (int e = threadIdx.x; e < n; e += NT) {
        const int es = (e & ~(S0 - 1)) | ((e + 1) & (S0 - 1));  // same row, next column
        for (int k = 0; k < K; ++k) {
          p[k * n + e] = __ldg(im1 + e * K + k);
          p[D + k * n + e] = __ldg(im2 + e * K + k);
          p[2 * D + k * n + e] = __ldg(im2 + es * K + k);
        }
      }
    }
    float* v = p + (sgi == 0 ? K * n : 0);
    for (int k = 0; k < nc; ++k, ++l, v += n) {
      const float* a = g1 + pg.var_off[l];
      const float* b = g2 + pg.var_off[l];
      for (int e = threadIdx.x; e < n; e += NT) {
        const int es = (e & ~(S - 1)) | ((e + 1) & (S - 1));
        const float va = __ldg(a + e), vb = __ldg(b + e);
        v[e] = va;
        v[D + e] = vb;
        v[2 * D + e] = __ldg(b + es);
        one_root = one_root && one_root_var(va) && one_root_var(vb);
      }
    }
    p += 3 * D;
  }
  cx.K = K;
  cx.inv_k = 1.f / (float)K;
  cx.acc_q = cx.acc_t = 0.f;
  cx.readout = pg.readout;
  return p;
}

// The lines of one pair that lines `first` .. `last` of its last segment take (two more on
// each side per segment before): those of segment 0, each completed pooled line right after
// the last of its three. Barriers only between lines: the threads that take a pooled line
// (the first 128, the first 32) do so while the others are at the next line of segment 0, and
// the line after that, which overwrites the slots just read, starts behind a barrier.
// NSEG > 0: segment count and conv counts N1, N2 fixed at compile time (the common
// Myrtle shapes), so that only the code this network runs is in the kernel.
template <int N0, int NSEG, int N1, int N2, int RO, bool ROOTS, int COMP, int KC>
__device__ __forceinline__ void chain_lines(ChainCtx& cx, const ntg_chain_t& pg, int nseg,
                                            float* const (&sec)[3], float* slots, int first,
                                            int last) {
  const int nc1 = NSEG > 0 ? (NSEG > 1 ? N1 : 0) : (nseg > 1 ? pg.nconv[1] : 0);
  const int nc2 = NSEG > 0 ? (NSEG > 2 ? N2 : 0) : (nseg > 2 ? pg.nconv[2] : 0);
  float* slots2 = slots + kSlots1;
  // lines of segments 1 and 0 that are taken
  int f1 = first, l1 = last;
  if (nseg > 2) {
    f1 = max(2 * first - 1, -(S1 - 1));
    l1 = min(2 * last + 1, S1 - 1);
  }
  const int f0 = nseg > 1 ? max(2 * f1 - 1, -(S0 - 1)) : first;
  const int l0 = nseg > 1 ? min(2 * l1 + 1, S0 - 1) : last;
  for (int d0 = f0; d0 <= l0; ++d0) {
    if (nseg == 1) {
      chain_line<S0, N0, true, true, RO, ROOTS, COMP, KC>(cx, pg, 0, sec[0], nullptr, nullptr, d0);
      continue;
    }
    chain_line<S0, N0, true, false, RO, ROOTS, COMP, KC>(cx, pg, 0, sec[0], nullptr, slots, d0);
    __syncthreads();
    const int m1 = (d0 - 1) / 2;
    if (!(d0 & 1) || m1 < f1) continue;
    if (nseg == 2) {
      pooled_line<S1, true, NSEG == 2 ? N1 : -1, RO, ROOTS, COMP>(cx, pg, nc1, N0, sec[1], slots,
                                                                  nullptr, m1);
      continue;
    }
    pooled_line<S1, false, NSEG == 3 ? N1 : -1, RO, ROOTS, COMP>(cx, pg, nc1, N0, sec[1], slots,
                                                                 slots2, m1);
    const int m2 = (m1 - 1) / 2;
    if (!(m1 & 1) || m2 < first) continue;
    if (threadIdx.x < 8 * S1) {  // the threads of segment 1: its three lines are in
      asm volatile("bar.sync 1, %0;" ::"n"(8 * S1) : "memory");
      pooled_line<S2, true, NSEG == 3 ? N2 : -1, RO, ROOTS, COMP>(cx, pg, nc2, N0 + nc1, sec[2],
                                                                  slots2, nullptr, m2);
    }
  }
}

// The readout's divisor and where a pair's two results go.
__device__ __forceinline__ void chain_write(const ntg_chain_t& pg, float sq, float st,
                                            float* out_q, float* out_t, int64_t o1, int64_t o2) {
  const int Sl = S0 >> (pg.nseg - 1);
  const float cnt = pg.readout == 0 ? (float)Sl * Sl * Sl * Sl : (float)Sl * Sl;
  out_q[o1] = sq / cnt;
  if (out_t) out_t[o1] = st / cnt;
  if (o2 >= 0) {
    out_q[o2] = sq / cnt;
    if (out_t) out_t[o2] = st / cnt;
  }
}

__device__ __forceinline__ void chain_place(const ChainGrid& g, int64_t pair, int64_t& gi,
                                            int64_t& gj, int64_t& o1, int64_t& o2) {
  int64_t i, j;
  if (g.sym == 1) {
    tri_pair(pair, g.n1, i, j);
  } else if (g.sym == 3) {
    i = j = pair;
  } else {
    i = pair / g.n2;
    j = pair - i * g.n2;
  }
  gi = g.r0 + i;
  gj = (g.sym == 3 ? g.r0 : g.c0) + j;
  o1 = g.sym == 3 ? i : g.sym ? gi * g.ld_out + gj : i * g.ld_out + j;
  o2 = (g.sym == 1 || g.sym == 2) && gi != gj ? gj * g.ld_out + gi : -1;
}

template <int N0, int NSEG, int N1, int N2, int RO, int COMP, int KC>
__device__ __forceinline__ void chain_pair(const ntg_chain_t& pg, const float* __restrict__ x1,
                                           const float* __restrict__ x2, int64_t gi, int64_t gj,
                                           const float* __restrict__ var1,
                                           const float* __restrict__ var2, float* slots,
                                           int first, int last, float* sums,
                                           float* __restrict__ out_q, float* __restrict__ out_t,
                                           int64_t o1, int64_t o2) {
  extern __shared__ __align__(16) float smem[];
  const int nseg = NSEG > 0 ? NSEG : pg.nseg;
  const int64_t im = (int64_t)S0 * S0 * pg.channels;
  ChainCtx cx;
  float* sec[3] = {nullptr, nullptr, nullptr};
  bool one_root = true;
  float* red = load_pair(cx, pg, nseg, x1 + gi * im, x2 + gj * im, var1 + gi * pg.var_stride,
                         var2 + gj * pg.var_stride, smem, sec, one_root);  // 2 * NT / 32 floats
  one_root = __syncthreads_and(one_root);
  auto lines = [&](auto two_roots) {
    chain_lines<N0, NSEG, N1, N2, RO, decltype(two_roots)::value, COMP, KC>(cx, pg, nseg, sec,
                                                                            slots, first, last);
  };
  if constexpr (RO == 1) {
    if (one_root) lines(std::false_type());
    else lines(std::true_type());
  } else {
    lines(std::true_type());
  }

  // block reduction of the readout sums
  float aq = cx.acc_q, at = cx.acc_t;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    aq += __shfl_xor_sync(0xffffffffu, aq, o);
    at += __shfl_xor_sync(0xffffffffu, at, o);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red[warp] = aq;
    red[NT / 32 + warp] = at;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float sq = 0.f, st = 0.f;
    for (int w = 0; w < NT / 32; ++w) {
      sq += red[w];
      st += red[NT / 32 + w];
    }
    if (sums) {
      sums[0] = sq;
      sums[1] = st;
    } else {
      chain_write(pg, sq, st, out_q, out_t, o1, o2);
    }
  }
}

// Two CTAs per SM, each striding over the pairs. sym == 0: the pairs (r0 + i, c0 + j) of
// x1 x x2, result at out[i * ld + j] (out points at the tile). sym == 1: the pairs i <= j of
// the square tile of x1 with itself (r0 == c0, n1 == n2); sym == 2: all pairs of a tile of x1
// with itself whose row and column ranges are disjoint. For sym 1 and 2 out points at element
// (0, 0) of the whole kernel and each result is written at (gi, gj) and (gj, gi). sym == 3:
// the pairs (r0 + i, r0 + i) of x1 with itself, result at out[i]. slots: kSlotFloats of
// scratch per CTA (the pooled lines, kept in L2 so that two CTAs fit an SM).
template <int N0, int NSEG = 0, int N1 = 0, int N2 = 0, int RO = 0, int COMP = -1,
          int KC = 0>
__global__ void __launch_bounds__(NT, kChainCtasPerSm)
    chain_fwd_kernel(const __grid_constant__ ntg_chain_t pg, const float* __restrict__ x1,
                     const float* __restrict__ x2, const ChainGrid grid,
                     const float* __restrict__ var1, const float* __restrict__ var2,
                     float* __restrict__ out_q, float* __restrict__ out_t, float* slots,
                     const __grid_constant__ ChainParts parts) {
  float* mine = slots + blockIdx.x * kSlotFloats;
  for (int64_t item = blockIdx.x; item < grid.total * parts.n; item += gridDim.x) {
    const int64_t pair = item / parts.n;
    const int part = (int)(item - pair * parts.n);
    int64_t gi, gj, o1, o2;
    chain_place(grid, pair, gi, gj, o1, o2);
    chain_pair<N0, NSEG, N1, N2, RO, COMP, KC>(
        pg, x1, x2, gi, gj, var1, var2, mine, parts.first[part], parts.last[part],
        parts.n > 1 ? parts.sums + 2 * item : nullptr, out_q, out_t, o1, o2);
    __syncthreads();  // the next pair overwrites the images and maps
  }
}

// Runs the variances of a segment through its layers: d [S x S] in shared memory holds the
// spatial diagonal of a self pair's kernel before the segment and after it on return, tmp is
// scratch. A self pair's diagonal only couples to itself under the conv rule, and the entries
// are evaluated exactly as chain_line evaluates row 0 of line 0, so that the pair (i, i) has
// var1 var2 - q^2 == 0 there. Each layer's pre-activation variances go to the segment's
// sections and to `out`; one_root: see load_pair.
template <int RO>
__device__ __forceinline__ void diag_layers(const ntg_chain_t& pg, int S, int nc, int lbase,
                                            float* sec, int K, float* d, float* tmp, float* out,
                                            bool& one_root) {
  const int n = S * S, D = (K + nc) * n;
  for (int k = 0; k < nc; ++k) {
    const ntg_affine_t& af = pg.aff[lbase + k];
    const ActC ac = act_consts(pg.act[lbase + k]);
    float* v = sec + (K + k) * n;
    for (int e = threadIdx.x; e < n; e += NT)
      tmp[e] = ((e >= S ? d[e - S] : 0.f) + d[e]) + (e + S < n ? d[e + S] : 0.f);
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += NT) {
      const int w = e & (S - 1);
      const float c = fmaf(w + 1 < S ? 1.f : 0.f, w + 1 < S ? tmp[e + 1] : 0.f,
                           fmaf(w > 0 ? 1.f : 0.f, w > 0 ? tmp[e - 1] : 0.f, tmp[e]));
      float q = fmaf(af.w2 * (1.f / 9.f), c, af.b2);
      v[e] = v[D + e] = q;
      v[2 * D + (e & ~(S - 1)) + ((w + S - 1) & (S - 1))] = q;
      out[pg.var_off[lbase + k] + e] = q;
      one_root = one_root && one_root_var(q);
      if (ac.kind != NTG_ACT_NONE) {
        float t = 0.f;
        const float vi = q, sv = sqrt_var(q);
        act_apply<RO == 2>(ac, q, t, vi, vi, sv, sv);
      }
      d[e] = q;
    }
    __syncthreads();
  }
}

// The variance maps of every layer, one CTA per sample at a time (the samples of x1, then
// those of x2): segment 0's from the image alone; segment 1's from the diagonal of pooled line
// 0, which takes lines -1 .. 1; segment 2's from pooled line 0 of segment 1, which takes lines
// -3 .. 3: at most 10 of the 63 lines of the pair (i, i), nngp only, in one launch. (The
// materialised rules evaluate the whole per-sample kernel layer by layer: two launches and
// 12 MB of HBM per 32 x 32 layer and sample: 31 launches and 1.66 ms for the 120 samples of a
// Myrtle-5 K(x, x), against 0.2 ms.)
template <int N0, int RO, int KC>
__global__ void __launch_bounds__(NT, kChainCtasPerSm)
    chain_var_kernel(const __grid_constant__ ntg_chain_t pg, const float* __restrict__ x1,
                     int64_t n1, float* __restrict__ var1, const float* __restrict__ x2,
                     int64_t n2, float* __restrict__ var2, float* slots) {
  extern __shared__ __align__(16) float smem[];
  const int K = pg.channels, nseg = pg.nseg;
  const int nc1 = nseg > 1 ? pg.nconv[1] : 0, nc2 = nseg > 2 ? pg.nconv[2] : 0;
  float* mine = slots + blockIdx.x * kSlotFloats;
  float* sec[3];
  sec[0] = smem;
  sec[1] = sec[0] + 3 * (K + N0) * S0 * S0;
  sec[2] = sec[1] + 3 * nc1 * S1 * S1;
  float* d = sec[2] + 3 * nc2 * S2 * S2;  // [2][S0 * S0]
  float* tmp = d + S0 * S0;
  ChainCtx cx;
  cx.K = K;
  cx.inv_k = 1.f / (float)K;
  cx.acc_q = cx.acc_t = 0.f;
  cx.readout = pg.readout;
  for (int64_t i = blockIdx.x; i < n1 + n2; i += gridDim.x) {
    const float* im = i < n1 ? x1 + i * S0 * S0 * K : x2 + (i - n1) * S0 * S0 * K;
    float* out = i < n1 ? var1 + i * pg.var_stride : var2 + (i - n1) * pg.var_stride;
    const int D = (K + N0) * S0 * S0;
    for (int e = threadIdx.x; e < S0 * S0; e += NT) {
      const int es = (e & ~(S0 - 1)) | ((e + S0 - 1) & (S0 - 1));  // same row, column before
      float g = 0.f;
      for (int k = 0; k < K; ++k) {
        const float v = __ldg(im + e * K + k);
        sec[0][k * S0 * S0 + e] = v;
        sec[0][D + k * S0 * S0 + e] = v;
        sec[0][2 * D + k * S0 * S0 + es] = v;
        g = fmaf(v, v, g);
      }
      d[e] = g * cx.inv_k;
    }
    __syncthreads();
    // the spatial diagonal of pooled line 0 of a segment of size S: row 0 and its side row
    auto pooled_diag = [&](const float* slot, int S) {
      const int plane = (S + S / 2) * S;
      for (int e = threadIdx.x; e < S * S; e += NT) {
        const float* p = slot + (e / S) * plane + (e & (S - 1));
        d[e] = (__ldcg(p) + __ldcg(p + (S + S / 2 - 1) * S)) * 0.0625f;
      }
      __syncthreads();
    };
    bool one_root = true;
    diag_layers<RO>(pg, S0, N0, 0, sec[0], K, d, tmp, out, one_root);
    // lines -1 .. 1 of segment 0 for segment 1's maps, then -3 .. 3 with segment 1 as well
    // for segment 2's
    auto segments = [&](auto two_roots) {
      constexpr bool ROOTS = decltype(two_roots)::value;
      for (int stage = 1; stage < nseg; ++stage) {
        const int w = stage == 1 ? 1 : 3;
        for (int d0 = -w; d0 <= w; ++d0) {
          chain_line<S0, N0, true, false, RO, ROOTS, -1, KC, false>(cx, pg, 0, sec[0], nullptr,
                                                                    mine, d0);
          __syncthreads();
          if (stage == 2 && (d0 & 1) && d0 > -3)
            pooled_line<S1, false, -1, RO, ROOTS, -1, false>(cx, pg, nc1, N0, sec[1], mine,
                                                             mine + kSlots1, (d0 - 1) / 2);
        }
        if (stage == 2) __syncthreads();
        pooled_diag(stage == 1 ? mine : mine + kSlots1, S0 >> stage);
        diag_layers<RO>(pg, S0 >> stage, stage == 1 ? nc1 : nc2, stage == 1 ? N0 : N0 + nc1,
                        sec[stage], 0, d, tmp, out, one_root);
      }
    };
    // By the rule of a pair of this sample (chain_pair), which goes by all maps, or
    // var1 var2 - q^2 would not be 0 in the pair: the pooled variances are sums over entries that
    // the two forms round differently.
    bool roots = RO != 1 || !__syncthreads_and(one_root);
    if constexpr (RO == 1) {
      if (!roots) {
        segments(std::false_type());
        roots = !__syncthreads_and(one_root);
      }
    }
    if (roots) segments(std::true_type());
  }
}

template <int N0, int RO, int KC = 0>
cudaError_t launch_var_k(const ntg_chain_t& pg, const VarArgs& a) {
  const size_t sm = chain_smem_bytes(pg) + 2 * S0 * S0 * sizeof(float);
  auto kernel = chain_var_kernel<N0, RO, KC>;
  cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  const int64_t n = a.n1 + a.n2;
  if (e == cudaSuccess)
    kernel<<<(unsigned)(n < kChainCtas ? n : kChainCtas), NT, sm, a.stream>>>(
        pg, a.x1, a.n1, a.var1, a.x2, a.n2, a.var2, a.slots);
  return e;
}

template <int N0, int NSEG, int N1, int N2, int RO = 0, int COMP = -1, int KC = 0>
cudaError_t launch_chain_k(const ntg_chain_t& pg, const ChainArgs& a) {
  const size_t sm = chain_smem_bytes(pg);
  auto kernel = chain_fwd_kernel<N0, NSEG, N1, N2, RO, COMP, KC>;
  cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e == cudaSuccess)
    kernel<<<(unsigned)a.ctas, NT, sm, a.stream>>>(pg, a.x1, a.x2, a.grid, a.var1, a.var2,
                                                   a.out_q, a.out_t, a.slots, a.parts);
  return e;
}

// The Myrtle shapes: kernels specialised to their segments; images of three channels with the
// ReLU family also to their precision (all layers share the precision of one call).
template <int N0, int N1, int N2>
cudaError_t launch_myrtle(bool relu_only, const ntg_chain_t& pg, const ChainArgs& a) {
  if (!relu_only) return launch_chain_k<N0, 3, N1, N2, 0>(pg, a);
  if (pg.channels != 3) return launch_chain_relu(pg, a);
  bool comp = false;
  for (int l = 0; l < NTG_CHAIN_MAX_LAYERS; ++l) comp = comp || pg.act[l].compensated != 0;
  return comp ? launch_chain_k<N0, 3, N1, N2, 1, 1, 3>(pg, a)
              : launch_chain_k<N0, 3, N1, N2, 1, 0, 3>(pg, a);
}

}  // namespace
}  // namespace ntg
