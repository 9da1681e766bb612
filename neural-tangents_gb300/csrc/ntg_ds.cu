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
// from the same code on every sample with itself, in a launch before. Bound by issue (76 % of
// the active slots; FP32 and shared memory about even): 100 x 90 pairs of 32 x 32 x 3 images
// through three 3 x 3 convs take 158 us (a third more with the window sizes read at run time),
// against 815 us in 27 launches for the layer rules, which move every layer's tensors through
// HBM.
//
// A network with poolings before its Flatten needs more than the diagonal, but not the whole
// (a c)^2 kernel: an entry of the readout sees the offsets (h' - h, w' - w) within k - 1 of the
// last pooling, those within s (k - 1) + k - 1 of the one before, and so on (convolutions of
// stride 1 keep an offset). For a fixed offset a layer is the same stencil on a plane of at
// most a x c entries, so the kernel walks the planes of the band one after another, the
// diagonal first (it gives a sample's variances), and adds each into the pooled planes of the
// next level in shared memory. One 2 x 2 pooling behind two convs on 28 x 28 images: 9 planes,
// 456 pairs in 57 us and the 43 samples' variances in 36 (a serial walk, few CTAs), against 5.8
// ms in 28 launches for the layer rules on 28^4 entries a pair.
#include <string>

#include "ntg_common.cuh"

namespace ntg {
namespace {

constexpr int kDsThreads = 256;

// The layers [first, last) between two poolings, and the planes (offsets |.| <= da, dc) of their
// input: a x c entries each, from the images or, behind a pooling, at acc.
struct DsLevel {
  int first, last, a, c, da, dc, acc;
};
struct DsBand {
  int nlevels, acc;  // entries of all pooled planes
  DsLevel level[NTG_DS_MAX_LAYERS + 1];
};

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
// layer. F: the window of every layer when it is F x F, 0: any windows. BAND: with poolings.
template <bool SELF, bool RELU, int F, bool BAND>
__global__ void __launch_bounds__(kDsThreads)
    ds_chain_kernel(const __grid_constant__ ntg_ds_chain_t pg, const __grid_constant__ DsBand band,
                    const DsGrid g) {
  extern __shared__ __align__(16) float smem[];
  const int P0 = pg.a * pg.c, K = pg.channels;
  constexpr bool MAPS = !SELF || BAND;  // the maps of sample 1 are read back
  // [K][P0] image 1 | layer maps of sample 1 | two planes of (nngp, ntk) | pooled planes |
  // reduction
  float* x1s = smem;
  float* v1s = x1s + K * P0;
  const int head = K * P0 + (MAPS ? pg.var_stride : 0);
  float2* A = reinterpret_cast<float2*>(smem + (head + 1) / 2 * 2);
  float2* B = A + pg.plane;
  float2* pooled = B + pg.plane;
  float* red = reinterpret_cast<float*>(pooled + (BAND ? band.acc : 0));
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
    if (BAND)
      for (int e = tid; e < band.acc; e += kDsThreads) pooled[e] = make_float2(0.f, 0.f);
    float sq = 0.f, st = 0.f;
    const int nlevels = BAND ? band.nlevels : 1;
    for (int lv = 0; lv < nlevels; ++lv) {
      const DsLevel& level = band.level[lv];
      const int first = BAND ? level.first : 0, end = BAND ? level.last : pg.nlayers;
      const int a0 = BAND ? level.a : pg.a, cc0 = BAND ? level.c : pg.c;
      const int da = BAND ? level.da : 0, dc = BAND ? level.dc : 0;
      const int wide = 2 * dc + 1, noff = (2 * da + 1) * wide;
      for (int o = 0; o < noff; ++o) {
        // the diagonal first, then the others in order; entry (r, c) of plane (dr, ds) is that
        // of positions (r, c) and (r + dr, c + ds), for both on the map
        const int at = o == 0 ? noff / 2 : o <= noff / 2 ? o - 1 : o;
        const int dr = BAND ? at / wide - da : 0, ds = BAND ? at - at / wide * wide - dc : 0;
        const int rlo = dr < 0 ? -dr : 0, rcut = dr > 0 ? dr : 0;
        const int wlo = ds < 0 ? -ds : 0, wcut = ds > 0 ? ds : 0;
        const float2* in = A;
        if (!BAND || lv == 0) {
          // input covariance, channel by channel (requirements.py:556-569)
          for (int r = rlo + ty; on && r < a0 - rcut; r += rows) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int e = r * cc0 + c0 + u, e2 = e + dr * cc0 + ds;
              if (c0 + u < wlo || c0 + u >= cc0 - wcut) continue;
              float s = 0.f;
              for (int k = 0; k < K; ++k)
                s = fmaf(x1s[k * P0 + e],
                         SELF ? x1s[k * P0 + e2] : __ldg(im2 + (int64_t)e2 * K + k), s);
              A[e] = make_float2(__fmul_rn(s, inv_k), 0.f);
            }
          }
        } else {
          in = pooled + level.acc + at * a0 * cc0;
        }
        __syncthreads();
        int a = a0, c = cc0;
        if (BAND && first == end) {  // a pooling right before the readout
          for (int e = tid; e < a * c; e += kDsThreads) {
            sq += in[e].x;
            st += in[e].y;
          }
        }
        for (int l = first; l < end; ++l) {
          const ntg_ds_layer_t& ly = pg.layer[l];
          const int ao = ly.ao, co = ly.co;
          const bool last = l + 1 == pg.nlayers && (!BAND || lv + 1 == nlevels);
          const bool ok0 = c0 >= wlo && c0 < co - wcut, ok1 = c0 + 1 >= wlo && c0 + 1 < co - wcut;
          // window sums along the columns, for every row of the input
          for (int r = rlo + ty; on && r < a - rcut; r += rows) {
            const float2* src = in + r * c;
            P2 h[2] = {p2s(0.f), p2s(0.f)};
            const int lo = c0 - ly.pw, fw = F ? F : ly.fw;
            // both windows in one walk: column lo + e is entry e of the first, e - 1 of the
            // second
#pragma unroll
            for (int e = 0; e <= fw; ++e) {
              const int cc = lo + e;
              P2 v = p2s(0.f);
              if (cc >= wlo && cc < c - wcut) v = p2ld(reinterpret_cast<const float*>(src + cc));
              if (e < fw) h[0] = add2(h[0], v);
              if (e > 0) h[1] = add2(h[1], v);
            }
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(B + r * co + c0);
            if (ok0) dst[0] = h[0].v;
            if (ok1) dst[1] = h[1].v;
          }
          __syncthreads();
          // along the rows, the affine rule and the activation
          const ActC ac = act_consts(ly.act);
          const float sc = 1.f / (float)(ly.fh * ly.fw);
          const float* v1m = v1s + ly.var_off;
          for (int r = rlo + ty; on && r < ao - rcut; r += rows) {
            if (!ok0 && !ok1) continue;
            P2 s[2] = {p2s(0.f), p2s(0.f)};
            const int fh = F ? F : ly.fh;
#pragma unroll
            for (int d = 0; d < fh; ++d) {
              const int rr = r + d - ly.ph;
              if (rr < rlo || rr >= a - rcut) continue;
              const float* src = reinterpret_cast<const float*>(B + rr * co + c0);
              if (ok0) s[0] = add2(s[0], p2ld(src));
              if (ok1) s[1] = add2(s[1], p2ld(src + 2));
            }
            float q[2], t[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              float cq, ct;
              p2u(s[u], cq, ct);
              apply_affine(ly.aff, cq, ct, !SELF, q[u], t[u], sc);
              if (SELF) t[u] = 0.f;
            }
            const int e = r * co + c0, e2 = e + dr * co + ds;
            if (ac.kind != NTG_ACT_NONE) {
              float v1[2] = {1.f, 1.f}, v2[2] = {1.f, 1.f};
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                if (!(u ? ok1 : ok0)) continue;
                if (SELF && (!BAND || o == 0)) {
                  v1[u] = v2[u] = q[u];
                  own[ly.var_off + e + u] = q[u];
                  if (BAND) v1s[ly.var_off + e + u] = q[u];
                } else {
                  v1[u] = v1m[e + u];
                  v2[u] = SELF ? v1m[e2 + u] : __ldg(v2m + ly.var_off + e2 + u);
                }
              }
              if (RELU) {
                P2 qq = p2(q[0], q[1]), tt = p2(t[0], t[1]);
                abrelu2_v<-1, true>(ac, qq, tt, p2(v1[0], v1[1]), p2(v2[0], v2[1]));
                p2u(qq, q[0], q[1]);
                p2u(tt, t[0], t[1]);
              } else {
#pragma unroll
                for (int u = 0; u < 2; ++u)
                  act_apply(ac, q[u], t[u], v1[u], v2[u], sqrt_var(v1[u]), sqrt_var(v2[u]));
              }
            }
            if (last) {
              sq += (ok0 ? q[0] : 0.f) + (ok1 ? q[1] : 0.f);
              st += (ok0 ? t[0] : 0.f) + (ok1 ? t[1] : 0.f);
            } else {
              if (ok0) A[e] = make_float2(q[0], t[0]);
              if (ok1) A[e + 1] = make_float2(q[1], t[1]);
            }
          }
          __syncthreads();
          in = A;
          a = ao;
          c = co;
        }
        if (BAND && lv + 1 < nlevels) {
          // Window sums of this plane for the planes of the next level that see it: position
          // r s + u of the first sample and (r + d) s + u' of the second, u' - u = dr - s d.
          // Each thread owns its entries.
          const ntg_ds_layer_t& ly = pg.layer[end - 1];
          const DsLevel& nx = band.level[lv + 1];
          for (int na = -nx.da; na <= nx.da; ++na) {
            const int ma = dr - ly.pool_sh * na;
            const int u0 = ma < 0 ? -ma : 0, u1 = ly.pool_h - (ma > 0 ? ma : 0);
            if (u0 >= u1) continue;
            for (int nc = -nx.dc; nc <= nx.dc; ++nc) {
              const int mc = ds - ly.pool_sw * nc;
              const int w0 = mc < 0 ? -mc : 0, w1 = ly.pool_w - (mc > 0 ? mc : 0);
              if (w0 >= w1) continue;
              float2* dst = pooled + nx.acc +
                            ((na + nx.da) * (2 * nx.dc + 1) + nc + nx.dc) * nx.a * nx.c;
              for (int e = tid; e < nx.a * nx.c; e += kDsThreads) {
                const int r = e / nx.c, w = e - r * nx.c;
                if (r + na < 0 || r + na >= nx.a || w + nc < 0 || w + nc >= nx.c) continue;
                P2 s = p2s(0.f);
                for (int u = u0; u < u1; ++u)
                  for (int x = w0; x < w1; ++x)
                    s = add2(s, p2ld(reinterpret_cast<const float*>(
                                    A + (r * ly.pool_sh + u) * c + w * ly.pool_sw + x)));
                float* d = reinterpret_cast<float*>(dst + e);
                const P2 v = fma2(s, p2s(ly.pool_scale), p2ld(d));
                *reinterpret_cast<unsigned long long*>(d) = v.v;
              }
            }
          }
          __syncthreads();
        }
      }
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

size_t ds_smem(const ntg_ds_chain_t& pg, const DsBand& band, bool self) {
  const bool maps = !self || band.nlevels > 1;
  const size_t f = (size_t)pg.channels * pg.a * pg.c + (maps ? pg.var_stride : 0);
  return sizeof(float) *
         ((f + 1) / 2 * 2 + 4 * (size_t)pg.plane + 2 * (size_t)band.acc + 2 * kDsThreads / 32);
}

template <bool SELF, bool BAND>
cudaError_t launch_ds(const ntg_ds_chain_t& pg, const DsBand& band, const DsGrid& g, bool relu,
                      bool three, int64_t blocks, cudaStream_t s) {
  auto kernel =
      three ? (relu ? ds_chain_kernel<SELF, true, 3, BAND> : ds_chain_kernel<SELF, false, 3, BAND>)
            : (relu ? ds_chain_kernel<SELF, true, 0, BAND> : ds_chain_kernel<SELF, false, 0, BAND>);
  const size_t sm = ds_smem(pg, band, SELF);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e == cudaSuccess) kernel<<<(unsigned)blocks, kDsThreads, sm, s>>>(pg, band, g);
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
  DsBand band{};
  band.nlevels = 1;
  band.level[0] = DsLevel{0, 0, a, c, 0, 0, 0};
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
    band.level[band.nlevels - 1].last = l + 1;
    if (ly.pool_h == 0) continue;
    // windows inside the map
    NTG_REQUIRE(ly.pool_h > 0 && ly.pool_w > 0 && ly.pool_h <= a && ly.pool_w <= c &&
                    ly.pool_sh > 0 && ly.pool_sw > 0,
                "ntg_ds_chain: bad pooling geometry");
    a = (a - ly.pool_h) / ly.pool_sh + 1;
    c = (c - ly.pool_w) / ly.pool_sw + 1;
    band.level[band.nlevels++] = DsLevel{l + 1, l + 1, a, c, 0, 0, 0};
  }
  // the offsets that the readout sees, from the last level back
  for (int v = band.nlevels - 2; v >= 0; --v) {
    DsLevel& lo = band.level[v];
    const DsLevel& hi = band.level[v + 1];
    const ntg_ds_layer_t& ly = pg.layer[lo.last - 1];
    const int da = ly.pool_sh * hi.da + ly.pool_h - 1, dc = ly.pool_sw * hi.dc + ly.pool_w - 1;
    lo.da = da < ly.ao - 1 ? da : ly.ao - 1;
    lo.dc = dc < ly.co - 1 ? dc : ly.co - 1;
  }
  int64_t acc = 0;
  for (int v = 1; v < band.nlevels; ++v) {
    DsLevel& lv = band.level[v];
    lv.acc = (int)acc;
    acc += (int64_t)(2 * lv.da + 1) * (2 * lv.dc + 1) * lv.a * lv.c;
    NTG_REQUIRE(acc < (1 << 20), "ntg_ds_chain: network needs more shared memory than a CTA has");
  }
  band.acc = (int)acc;
  NTG_REQUIRE(pg.var_stride == off, "ntg_ds_chain: var_stride does not fit the layers");
  NTG_REQUIRE(ds_smem(pg, band, false) <= 232448, "ntg_ds_chain: network needs more shared memory than a CTA has");
  const bool pools = band.nlevels > 1;
  cudaStream_t s = as_stream(stream);
  DsGrid g{x1, x2, n1, x2 ? n2 : 0, var1, var2, cov1, cov2, 0, 1, (pg.c + 1) / 2};
  cudaError_t e = pools ? launch_ds<true, true>(pg, band, g, relu, three, n1 + g.n2, s)
                        : launch_ds<true, false>(pg, band, g, relu, three, n1 + g.n2, s);
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
    e = pools ? launch_ds<false, true>(pg, band, g, relu, three, blocks, s)
              : launch_ds<false, false>(pg, band, g, relu, three, blocks, s);
    note_launch();
  }
  if (e != cudaSuccess)
    return fail(NTG_ERR_CUDA, std::string("ntg_ds_chain: ") + cudaGetErrorString(e));
  return check_launch("ntg_ds_chain");
}
