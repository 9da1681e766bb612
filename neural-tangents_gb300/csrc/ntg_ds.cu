// Whole-network kernel of conv networks on diagonal-spatial kernels (linear.py:3381-3437: the
// reference's form for conv nets whose readout only sees the spatial diagonal) on sm_103a.
//
// A pair's nngp and ntk are two planes of a x c entries. One CTA takes a sample of x1 and a run
// of samples of x2, keeps the x1 image and its variance maps in shared memory, and takes each
// pair from the input covariance through every Conv / Dense + activation layer to the mean of
// the positions, the planes never leaving the SM. Entries are (nngp, ntk) pairs in shared
// memory, so that one 8-byte access and one packed add serve both in the window sums, which
// run along the columns, then along the rows; a thread owns two neighbouring columns, so that
// the activation rule runs on packed pairs. The variances (elementwise on the diagonal) come
// from the same code on every sample with itself, in a launch before. Bound by issue (70 % of
// the slots; FP32 and shared memory about even): 100 x 90 pairs of 32 x 32 x 3 images through
// three 3 x 3 convs take 144 us (194 us with the window sizes read at run time), against 815
// us in 27 launches for the layer rules, which move every layer's tensors through HBM.
#include <string>

#include "ntg_common.cuh"

namespace ntg {
namespace {

constexpr int kDsThreads = 256;

struct DsGrid {
  const float *x1, *x2;
  int64_t n1, n2;
  float *var1, *var2;    // [N][layer maps] pre-activation variances
  float *out_q, *out_t;  // pairs: [N1, N2]; SELF: cov1 [N1], cov2 [N2]
  int sym;               // x2 == x1: the pairs i <= j, mirrored
  int run;               // samples of x2 per CTA
  int tx;                // threads along a row (two columns each)
};

// SELF: each sample with itself (those of x1, then of x2), nngp only: writes the variance maps
// and the readout; else pairs. RELU: an ABRelu without do_stabilize or no activation in every
// layer. F: the window of every layer when it is F x F, 0: any windows.
template <bool SELF, bool RELU, int F>
__global__ void __launch_bounds__(kDsThreads)
    ds_chain_kernel(const __grid_constant__ ntg_ds_chain_t pg, const DsGrid g) {
  extern __shared__ __align__(16) float smem[];
  const int P0 = pg.a * pg.c, K = pg.channels;
  // [K][P0] image 1 | layer maps of sample 1 | two planes of (nngp, ntk) | reduction
  float* x1s = smem;
  float* v1s = x1s + K * P0;
  const int head = K * P0 + (SELF ? 0 : pg.var_stride);
  float2* A = reinterpret_cast<float2*>(smem + (head + 1) / 2 * 2);
  float2* B = A + pg.plane;
  float* red = reinterpret_cast<float*>(B + pg.plane);
  const int tid = threadIdx.x;
  const int ty = tid / g.tx, c0 = 2 * (tid - ty * g.tx);
  const int rows = kDsThreads / g.tx;       // rows per pass
  const bool on = ty < rows;                // threads past the last whole row only synchronise
  const float inv_k = 1.f / (float)K;

  int64_t i, j0, j1;
  if (SELF) {
    i = blockIdx.x;
    j0 = 0;
    j1 = 1;
  } else {
    const int64_t runs = (g.n2 + g.run - 1) / g.run;
    i = blockIdx.x / runs;
    j0 = (blockIdx.x - i * runs) * g.run;
    j1 = j0 + g.run < g.n2 ? j0 + g.run : g.n2;
    if (g.sym && j0 < i) j0 = i;
    if (j0 >= j1) return;
  }
  const bool second = SELF && i >= g.n1;
  const int64_t n = second ? i - g.n1 : i;
  const float* im1 = (second ? g.x2 : g.x1) + n * (int64_t)P0 * K;
  float* own = (second ? g.var2 : g.var1) + n * pg.var_stride;
  for (int e = tid; e < P0; e += kDsThreads)
    for (int k = 0; k < K; ++k) x1s[k * P0 + e] = __ldg(im1 + (int64_t)e * K + k);
  if (!SELF)
    for (int e = tid; e < pg.var_stride; e += kDsThreads) v1s[e] = own[e];
  __syncthreads();

  for (int64_t j = j0; j < j1; ++j) {
    const float* im2 = g.x2 + j * (int64_t)P0 * K;
    const float* v2m = SELF ? nullptr : g.var2 + j * pg.var_stride;
    // input covariance, channel by channel (requirements.py:556-569)
    for (int r = ty; on && r < pg.a; r += rows) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = r * pg.c + c0 + u;
        if (c0 + u >= pg.c) continue;
        float s = 0.f;
        for (int k = 0; k < K; ++k) {
          const float x = x1s[k * P0 + e];
          s = fmaf(x, SELF ? x : __ldg(im2 + (int64_t)e * K + k), s);
        }
        A[e] = make_float2(__fmul_rn(s, inv_k), 0.f);
      }
    }
    __syncthreads();
    int a = pg.a, c = pg.c;
    float sq = 0.f, st = 0.f;
    for (int l = 0; l < pg.nlayers; ++l) {
      const ntg_ds_layer_t& ly = pg.layer[l];
      const int ao = ly.ao, co = ly.co;
      const bool last = l + 1 == pg.nlayers;
      // window sums along the columns, for every row of the input
      for (int r = ty; on && r < a; r += rows) {
        const float2* src = A + r * c;
        P2 h[2] = {p2s(0.f), p2s(0.f)};
        const int lo = c0 - ly.pw, fw = F ? F : ly.fw;
        // both windows in one walk: column lo + e is entry e of the first, e - 1 of the second
#pragma unroll
        for (int e = 0; e <= fw; ++e) {
          const int cc = lo + e;
          P2 v = p2s(0.f);
          if (cc >= 0 && cc < c) v = p2ld(reinterpret_cast<const float*>(src + cc));
          if (e < fw) h[0] = add2(h[0], v);
          if (e > 0) h[1] = add2(h[1], v);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (c0 + u < co)
            *reinterpret_cast<unsigned long long*>(B + r * co + c0 + u) = h[u].v;
      }
      __syncthreads();
      // along the rows, the affine rule and the activation
      const ActC ac = act_consts(ly.act);
      const float sc = 1.f / (float)(ly.fh * ly.fw);
      const float* v1m = v1s + ly.var_off;
      for (int r = ty; on && r < ao; r += rows) {
        if (c0 >= co) continue;
        const bool two = c0 + 1 < co;
        P2 s[2] = {p2s(0.f), p2s(0.f)};
        const int fh = F ? F : ly.fh;
#pragma unroll
        for (int d = 0; d < fh; ++d) {
          const int rr = r + d - ly.ph;
          if (rr < 0 || rr >= a) continue;
          const float* src = reinterpret_cast<const float*>(B + rr * co + c0);
          s[0] = add2(s[0], p2ld(src));
          if (two) s[1] = add2(s[1], p2ld(src + 2));
        }
        float q[2], t[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float cq, ct;
          p2u(s[u], cq, ct);
          apply_affine(ly.aff, cq, ct, !SELF, q[u], t[u], sc);
          if (SELF) t[u] = 0.f;
        }
        const int e = r * co + c0;
        if (ac.kind != NTG_ACT_NONE) {
          float v1[2], v2[2];
          if (SELF) {
            v1[0] = v2[0] = q[0];
            v1[1] = v2[1] = q[1];
            own[ly.var_off + e] = q[0];
            if (two) own[ly.var_off + e + 1] = q[1];
          } else {
            v1[0] = v1m[e];
            v2[0] = __ldg(v2m + ly.var_off + e);
            v1[1] = two ? v1m[e + 1] : v1[0];
            v2[1] = two ? __ldg(v2m + ly.var_off + e + 1) : v2[0];
          }
          if (RELU) {
            P2 qq = p2(q[0], q[1]), tt = p2(t[0], t[1]);
            abrelu2_v(ac, qq, tt, p2(v1[0], v1[1]), p2(v2[0], v2[1]));
            p2u(qq, q[0], q[1]);
            p2u(tt, t[0], t[1]);
          } else {
#pragma unroll
            for (int u = 0; u < 2; ++u)
              act_apply(ac, q[u], t[u], v1[u], v2[u], sqrt_var(v1[u]), sqrt_var(v2[u]));
          }
        }
        if (last) {
          sq += q[0] + (two ? q[1] : 0.f);
          st += t[0] + (two ? t[1] : 0.f);
        } else {
          A[e] = make_float2(q[0], t[0]);
          if (two) A[e + 1] = make_float2(q[1], t[1]);
        }
      }
      __syncthreads();
      a = ao;
      c = co;
    }
    // sum over the positions
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      st += __shfl_xor_sync(0xffffffffu, st, o);
    }
    if ((tid & 31) == 0) {
      red[tid >> 5] = sq;
      red[kDsThreads / 32 + (tid >> 5)] = st;
    }
    __syncthreads();
    if (tid == 0) {
      float fq = 0.f, ft = 0.f;
      for (int w = 0; w < kDsThreads / 32; ++w) {
        fq += red[w];
        ft += red[kDsThreads / 32 + w];
      }
      fq = fq / pg.divisor * pg.scale;
      ft = ft / pg.divisor * pg.scale;
      if (SELF) {
        (second ? g.out_t : g.out_q)[n] = fq;
      } else {
        g.out_q[i * g.n2 + j] = fq;
        if (g.out_t) g.out_t[i * g.n2 + j] = ft;
        if (g.sym && i != j) {
          g.out_q[j * g.n2 + i] = fq;
          if (g.out_t) g.out_t[j * g.n2 + i] = ft;
        }
      }
    }
    // the next pair's first barrier comes before red is written again
  }
}

size_t ds_smem(const ntg_ds_chain_t& pg, bool self) {
  const size_t f = (size_t)pg.channels * pg.a * pg.c + (self ? 0 : pg.var_stride);
  return sizeof(float) * ((f + 1) / 2 * 2 + 4 * (size_t)pg.plane + 2 * kDsThreads / 32);
}

template <bool SELF>
cudaError_t launch_ds(const ntg_ds_chain_t& pg, const DsGrid& g, bool relu, bool three,
                      int64_t blocks, cudaStream_t s) {
  auto kernel = three ? (relu ? ds_chain_kernel<SELF, true, 3> : ds_chain_kernel<SELF, false, 3>)
                      : (relu ? ds_chain_kernel<SELF, true, 0> : ds_chain_kernel<SELF, false, 0>);
  const size_t sm = ds_smem(pg, SELF);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e == cudaSuccess) kernel<<<(unsigned)blocks, kDsThreads, sm, s>>>(pg, g);
  return e;
}

}  // namespace
}  // namespace ntg

using namespace ntg;

extern "C" int ntg_ds_chain(void* stream, const ntg_ds_chain_t* prog, const float* x1,
                            const float* x2, int64_t n1, int64_t n2, float* var1, float* var2,
                            float* cov1, float* cov2, float* out_q, float* out_t) {
  NTG_REQUIRE(prog && x1 && var1 && cov1 && out_q, "ntg_ds_chain: null pointer");
  NTG_REQUIRE(!x2 == !var2 && !x2 == !cov2, "ntg_ds_chain: x2, var2 and cov2 go together");
  NTG_REQUIRE(n1 > 0 && (x2 ? n2 > 0 : n2 == n1), "ntg_ds_chain: bad sizes");
  ntg_ds_chain_t pg = *prog;
  NTG_REQUIRE(pg.nlayers > 0 && pg.nlayers <= NTG_DS_MAX_LAYERS, "ntg_ds_chain: bad layer count");
  NTG_REQUIRE(pg.a > 0 && pg.c > 0 && pg.c <= 2 * kDsThreads && pg.channels > 0 &&
                  pg.a <= 4096 && pg.channels <= 4096,
              "ntg_ds_chain: unsupported image size");
  int a = pg.a, c = pg.c, off = 0;
  bool relu = true, three = true;
  pg.plane = a * c;
  for (int l = 0; l < pg.nlayers; ++l) {
    ntg_ds_layer_t& ly = pg.layer[l];
    // stride 1 with zero padding: a window per output, at least one entry of it inside
    NTG_REQUIRE(ly.fh > 0 && ly.fw > 0 && ly.ph >= 0 && ly.pw >= 0 && ly.ph < ly.fh &&
                    ly.pw < ly.fw && ly.ao > 0 && ly.co > 0 && ly.ao <= a && ly.co <= c,
                "ntg_ds_chain: bad layer geometry");
    NTG_REQUIRE(ly.act.kind >= NTG_ACT_NONE && ly.act.kind <= NTG_ACT_GELU,
                "ntg_ds_chain: unknown activation kind");
    relu = relu && (ly.act.kind == NTG_ACT_NONE ||
                    (ly.act.kind == NTG_ACT_ABRELU && ly.act.stabilize <= 0.f));
    three = three && ly.fh == 3 && ly.fw == 3;
    NTG_REQUIRE(ly.var_off == off, "ntg_ds_chain: the layer maps follow one another");
    off += ly.ao * ly.co;
    if (a * ly.co > pg.plane) pg.plane = a * ly.co;
    a = ly.ao;
    c = ly.co;
  }
  NTG_REQUIRE(pg.var_stride == off, "ntg_ds_chain: var_stride does not fit the layers");
  NTG_REQUIRE(ds_smem(pg, false) <= 232448, "ntg_ds_chain: network needs more shared memory than a CTA has");
  cudaStream_t s = as_stream(stream);
  DsGrid g{x1, x2, n1, x2 ? n2 : 0, var1, var2, cov1, cov2, 0, 1, (pg.c + 1) / 2};
  cudaError_t e = launch_ds<true>(pg, g, relu, three, n1 + g.n2, s);
  note_launch();
  if (e == cudaSuccess) {
    g.sym = !x2;
    g.n2 = n2;
    g.out_q = out_q;
    g.out_t = out_t;
    if (g.sym) {
      g.x2 = x1;
      g.var2 = var1;
    }
    // samples of x2 per CTA: as many as leave eight CTAs per SM to balance with, so that the
    // image and maps of the x1 sample are loaded once for up to 16 pairs
    int64_t run = n1 * n2 / (152 * 8);
    g.run = (int)(run < 1 ? 1 : run > 16 ? 16 : run);
    const int64_t blocks = n1 * ceil_div(n2, g.run);
    NTG_REQUIRE(blocks < (1ll << 31), "ntg_ds_chain: grid too large");
    e = launch_ds<false>(pg, g, relu, three, blocks, s);
    note_launch();
  }
  if (e != cudaSuccess)
    return fail(NTG_ERR_CUDA, std::string("ntg_ds_chain: ") + cudaGetErrorString(e));
  return check_launch("ntg_ds_chain");
}
