// Flat (fully connected) inputs on sm_103a: the FP32 Gram x1 x2^T / D on CUDA cores and
// the per-sample variances, every entry one fmaf chain in ascending D, so that a variance
// equals the Gram's diagonal entry bit for bit whatever tile computed it.
#include <string>

#include "ntg_common.cuh"

namespace ntg {
namespace {

// Row-major lower triangle of tiles: t = i (i + 1) / 2 + j, j <= i.
__device__ __forceinline__ void tri_tile(int64_t t, int64_t& ti, int64_t& tj) {
  ti = (int64_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (ti * (ti + 1) / 2 > t) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  tj = t - ti * (ti + 1) / 2;
}

// ---------------------------------------------------------------------------
// Large Grams: 128 x 128 output tile per CTA, 16 x 16 threads, 8 x 8 outputs per thread
// (rows 4 ty + u and 64 + 4 ty + u, columns likewise in tx) read from shared memory as
// 16-byte words. Bound by FP32 issue: two columns are one packed fma.rn.f32x2 (each lane
// rounds as fmaf does), and the next 16-deep slice is loaded into registers while the
// current one is multiplied, so a slice costs one barrier and no exposed load latency.
// X X^T of [4096, 3072]: 1213 us (scalar fmaf, single buffer: 1383 us).
// SYM (x1 == x2): the tiles on or below the diagonal only, each off-diagonal one also
// stored transposed: fmaf(a, b, c) == fmaf(b, a, c), so the mirror is exactly the value
// the tile (j, i) would hold. VEC: d a multiple of 4 and both inputs 16-byte aligned.
// ---------------------------------------------------------------------------
template <bool SYM, bool VEC>
__global__ void __launch_bounds__(256, 2)
    gram_simt_kernel(const float* __restrict__ x1, const float* __restrict__ x2, int64_t n1,
                     int64_t n2, int64_t d, float inv_d, float* __restrict__ out) {
  constexpr int P = 128 + 4;
  __shared__ __align__(16) float As[2][16][P];
  __shared__ __align__(16) float Bs[2][16][P];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int64_t ti = blockIdx.y, tj = blockIdx.x;
  if (SYM) tri_tile(blockIdx.x, ti, tj);
  const int64_t row0 = ti * 128, col0 = tj * 128;
  // this thread's part of a slice: 8 consecutive k of one row (VEC: two 16-byte loads; a
  // row of 16 k is two threads), or 8 rows at one k
  float ra[8], rb[8];
  auto fetch = [&](int64_t k0) {
    if (VEC) {
      const int r = threadIdx.x >> 1;
      const int64_t gk = k0 + 8 * (threadIdx.x & 1);
      const int64_t gi = row0 + r, gj = col0 + r;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool in = gk + 4 * h < d;
        const float4 a = in && gi < n1
                             ? __ldg(reinterpret_cast<const float4*>(x1 + gi * d + gk + 4 * h))
                             : z;
        const float4 b = in && gj < n2
                             ? __ldg(reinterpret_cast<const float4*>(x2 + gj * d + gk + 4 * h))
                             : z;
        ra[4 * h] = a.x; ra[4 * h + 1] = a.y; ra[4 * h + 2] = a.z; ra[4 * h + 3] = a.w;
        rb[4 * h] = b.x; rb[4 * h + 1] = b.y; rb[4 * h + 2] = b.z; rb[4 * h + 3] = b.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int idx = threadIdx.x + 256 * e;
        const int r = idx >> 4;
        const int64_t gk = k0 + (idx & 15), gi = row0 + r, gj = col0 + r;
        ra[e] = (gi < n1 && gk < d) ? __ldg(x1 + gi * d + gk) : 0.f;
        rb[e] = (gj < n2 && gk < d) ? __ldg(x2 + gj * d + gk) : 0.f;
      }
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int idx = threadIdx.x + 256 * e;
      const int kk = VEC ? 8 * (threadIdx.x & 1) + e : idx & 15;
      const int r = VEC ? threadIdx.x >> 1 : idx >> 4;
      As[buf][kk][r] = ra[e];
      Bs[buf][kk][r] = rb[e];
    }
  };
  P2 acc[8][4];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = p2s(0.f);
  fetch(0);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = 0; k0 < d; k0 += 16) {
    const bool more = k0 + 16 < d;
    if (more) fetch(k0 + 16);
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][4 * ty]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][64 + 4 * ty]);
      const float* br = &Bs[buf][kk][4 * tx];
      const P2 b[4] = {p2ld(br), p2ld(br + 2), p2ld(br + 64), p2ld(br + 66)};
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const P2 au = p2s(a[u]);
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fma2(au, b[v], acc[u][v]);
      }
    }
    if (more) put(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  const bool vec = (n2 & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  const bool mirror = SYM && ti != tj;
  float r[8][8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      p2u(acc[u][v], r[u][2 * v], r[u][2 * v + 1]);
      r[u][2 * v] *= inv_d;
      r[u][2 * v + 1] *= inv_d;
    }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int64_t gi = row0 + (u < 4 ? 4 * ty + u : 64 + 4 * ty + u - 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t gj = col0 + 64 * h + 4 * tx;
      if (gi >= n1) continue;
      if (vec && gj + 3 < n2) {
        *reinterpret_cast<float4*>(out + gi * n2 + gj) =
            make_float4(r[u][4 * h], r[u][4 * h + 1], r[u][4 * h + 2], r[u][4 * h + 3]);
      } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (gj + v < n2) out[gi * n2 + gj + v] = r[u][4 * h + v];
      }
    }
  }
  if (mirror) {  // out[gj][gi] = tile[gi][gj]
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int64_t gj = col0 + (v < 4 ? 4 * tx + v : 64 + 4 * tx + v - 4);
      if (gj >= n1) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t gi = row0 + 64 * h + 4 * ty;
        if (vec && gi + 3 < n1) {
          *reinterpret_cast<float4*>(out + gj * n2 + gi) =
              make_float4(r[4 * h][v], r[4 * h + 1][v], r[4 * h + 2][v], r[4 * h + 3][v]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (gi + u < n1) out[gj * n2 + gi + u] = r[4 * h + u][v];
        }
      }
    }
  }
}

// 16- or 4-byte asynchronous copy to shared memory; `in` false writes zeros.
template <bool VEC>
__device__ __forceinline__ void cp_async(float* dst, const float* src, bool in) {
  const int n = in ? (VEC ? 16 : 4) : 0;
  if (VEC)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Rows [r0, r0 + ROWS) x columns [k0, k0 + BK) of x [n, d] into dst [ROWS][BK + 4].
template <int ROWS, int BK, int THREADS, bool VEC>
__device__ __forceinline__ void stage_rows(float* dst, const float* x, int64_t n, int64_t d,
                                           int64_t r0, int64_t k0) {
  constexpr int W = VEC ? 4 : 1, PER = BK / W;
#pragma unroll
  for (int e = 0; e < ROWS * PER / THREADS; ++e) {
    const int idx = threadIdx.x + THREADS * e;
    const int r = idx / PER, k = (idx % PER) * W;
    const bool in = r0 + r < n && k0 + k < d;  // VEC: d is a multiple of 4
    cp_async<VEC>(dst + r * (BK + 4) + k, in ? x + (r0 + r) * d + k0 + k : x, in);
  }
}

// ---------------------------------------------------------------------------
// Small Grams, which a 128-wide tile would leave on a few SMs: T x T output tile per CTA,
// each thread RU x RV outputs (rows ty + TY u, columns tx + 16 v) from
// k-contiguous shared rows read as 16-byte words, slices streamed by a 4-stage cp.async
// ring (one barrier per slice). The k order is that of gram_simt_kernel. Bound by the
// chain of D / BK slices per tile: 256 x 256 x 784 takes 12.4 us (128-wide tiles: 102 us).
// ---------------------------------------------------------------------------
template <int T, int BK, int RU, int RV, bool SYM, bool VEC>
__global__ void __launch_bounds__(16 * (T / RU))
    gram_small_kernel(const float* __restrict__ x1, const float* __restrict__ x2, int64_t n1,
                      int64_t n2, int64_t d, float inv_d, float* __restrict__ out) {
  constexpr int ST = 4, P = BK + 4, TY = T / RU, THREADS = 16 * TY;
  static_assert(16 * RV == T, "columns tx + 16 v cover the tile");
  __shared__ __align__(16) float As[ST][T * P];
  __shared__ __align__(16) float Bs[ST][T * P];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int64_t ti = blockIdx.y, tj = blockIdx.x;
  if (SYM) tri_tile(blockIdx.x, ti, tj);
  const int64_t row0 = ti * T, col0 = tj * T;
  const int64_t nk = (d + BK - 1) / BK;
  auto stage = [&](int64_t s) {
    if (s < nk) {
      stage_rows<T, BK, THREADS, VEC>(As[s % ST], x1, n1, d, row0, s * BK);
      stage_rows<T, BK, THREADS, VEC>(Bs[s % ST], x2, n2, d, col0, s * BK);
    }
    cp_commit();
  };
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) stage(s);
  float acc[RU][RV];
#pragma unroll
  for (int u = 0; u < RU; ++u)
#pragma unroll
    for (int v = 0; v < RV; ++v) acc[u][v] = 0.f;
  for (int64_t s = 0; s < nk; ++s) {
    cp_wait<ST - 2>();
    __syncthreads();  // slice s is in; slice s - 1 is done with, its slot is free
    stage(s + ST - 1);
    const float* A = As[s % ST] + ty * P;
    const float* B = Bs[s % ST] + tx * P;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      float4 a[RU], b[RV];
#pragma unroll
      for (int u = 0; u < RU; ++u) a[u] = *reinterpret_cast<const float4*>(A + TY * u * P + k);
#pragma unroll
      for (int v = 0; v < RV; ++v) b[v] = *reinterpret_cast<const float4*>(B + 16 * v * P + k);
#pragma unroll
      for (int u = 0; u < RU; ++u)
#pragma unroll
        for (int v = 0; v < RV; ++v) {
          float c = acc[u][v];
          c = fmaf(a[u].x, b[v].x, c);
          c = fmaf(a[u].y, b[v].y, c);
          c = fmaf(a[u].z, b[v].z, c);
          acc[u][v] = fmaf(a[u].w, b[v].w, c);
        }
    }
  }
  const bool mirror = SYM && ti != tj;
#pragma unroll
  for (int u = 0; u < RU; ++u)
#pragma unroll
    for (int v = 0; v < RV; ++v) {
      const int64_t gi = row0 + ty + TY * u, gj = col0 + tx + 16 * v;
      if (gi >= n1 || gj >= n2) continue;
      const float o = acc[u][v] * inv_d;
      out[gi * n2 + gj] = o;
      if (mirror) out[gj * n2 + gi] = o;
    }
}

// Per-row sum(x^2) / D, the Gram's chain along the diagonal: 32 rows per CTA streamed
// through a 4-stage cp.async ring by 128 threads, one lane of warp 0 per row running its
// chain (bound by the 4-cycle dependent fmaf: 4001 + 1999 rows of D = 3072 take 24 us; a
// thread per row reading global memory took 414 us). Blocks past the first input's rows
// take the second's (n2 == 0: none).
template <bool VEC>
__global__ void __launch_bounds__(128)
    cov_diag_kernel(const float* __restrict__ x1, int64_t n1, const float* __restrict__ x2,
                    int64_t n2, int64_t d, float inv_d, float* __restrict__ cov1,
                    float* __restrict__ cov2) {
  constexpr int ST = 4, BK = 64, P = BK + 4;
  __shared__ __align__(16) float Xs[ST][32 * P];
  const int64_t nb1 = (n1 + 31) / 32;
  const bool second = (int64_t)blockIdx.x >= nb1;
  const float* x = second ? x2 : x1;
  const int64_t n = second ? n2 : n1;
  const int64_t r0 = 32 * (second ? blockIdx.x - nb1 : blockIdx.x);
  const int64_t nk = (d + BK - 1) / BK;
  auto stage = [&](int64_t s) {
    if (s < nk) stage_rows<32, BK, 128, VEC>(Xs[s % ST], x, n, d, r0, s * BK);
    cp_commit();
  };
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) stage(s);
  float acc = 0.f;
  for (int64_t s = 0; s < nk; ++s) {
    cp_wait<ST - 2>();
    __syncthreads();
    stage(s + ST - 1);
    if (threadIdx.x < 32) {
      const float* p = Xs[s % ST] + threadIdx.x * P;
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        const float4 v = *reinterpret_cast<const float4*>(p + k);
        acc = fmaf(v.x, v.x, acc);
        acc = fmaf(v.y, v.y, acc);
        acc = fmaf(v.z, v.z, acc);
        acc = fmaf(v.w, v.w, acc);
      }
    }
  }
  if (threadIdx.x < 32 && r0 + threadIdx.x < n)
    (second ? cov2 : cov1)[r0 + threadIdx.x] = acc * inv_d;
}

// ---------------------------------------------------------------------------
// A run of Dense / activation rules on flat kernels in one pass: nngp and ntk are read
// once and written once however many layers the run has, and the per-sample kernels
// follow along. A CTA takes a 32 x 64 tile: 96 threads first run the variances of its
// rows and columns through the layers (the activation rule on a sample with itself, as
// affine_act_kernel evaluates it on a per-sample kernel) and leave each layer's
// pre-activation variance and its square root in shared memory; then every thread runs
// 8 entries (rows 4 warp + u, columns lane + 32 h) through them. Same operations per entry and per variance as one affine_act_kernel per
// layer, so the results are those bit for bit. Bound by FP32 issue for a large kernel, by
// the launch for a small one: three Erf layers of 4001 x 1999 take 65 us (18 launches,
// seven of them over nngp and ntk: 337 us), two ReLU layers of 256 x 256 4.1 us (29 us).
// ---------------------------------------------------------------------------
constexpr int kFlatRows = 32, kFlatCols = 64, kFlatSamples = kFlatRows + kFlatCols;

struct FlatRun {
  int n;
  ntg_flat_layer_t layer[NTG_FLAT_MAX_LAYERS];
};

// RELU: no activation or the ABRelu family without do_stabilize in every layer.
template <bool RELU>
__global__ void __launch_bounds__(256)
    flat_rules_kernel(const __grid_constant__ FlatRun run, const float* in_q, const float* in_t,
                      int64_t n1, int64_t n2, const float* var1, int64_t s1, const float* var2,
                      int64_t s2, float* out_q, float* out_t, float* cov1, float* cov2) {
  extern __shared__ float fv[];  // [layer][v | sqrt v][row or column]
  const int64_t ntx = (n2 + kFlatCols - 1) / kFlatCols;
  const int64_t by = blockIdx.x / ntx, bx = blockIdx.x - by * ntx;
  const int64_t r0 = by * kFlatRows, c0 = bx * kFlatCols;
  const int tid = threadIdx.x;
  if (tid < kFlatSamples) {
    const bool row = tid < kFlatRows;
    const int64_t i = row ? r0 + tid : c0 + tid - kFlatRows;
    const bool in = i < (row ? n1 : n2);
    float v = in ? (row ? var1[i * s1] : var2[i * s2]) : 0.f;
    for (int l = 0; l < run.n; ++l) {
      const ntg_flat_layer_t& ly = run.layer[l];
      if (ly.has_affine) v = fmaf(ly.aff.w2, v, ly.aff.b2);
      if (ly.act.kind != NTG_ACT_NONE) {
        const float s = sqrt_var(v);
        fv[(2 * l) * kFlatSamples + tid] = v;
        fv[(2 * l + 1) * kFlatSamples + tid] = s;
        const ActC ac = act_consts(ly.act);
        float t = 0.f;
        const float vi = v;
        act_apply<!RELU, !RELU>(ac, v, t, vi, vi, s, s);
      }
    }
    if (in && row && bx == 0 && cov1) cov1[i] = v;
    if (in && !row && by == 0 && cov2) cov2[i] = v;
  }
  __syncthreads();
  const int lane = tid & 31, w = 4 * (tid >> 5);
  float q[2][4], t[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = r0 + w + u, j = c0 + lane + 32 * h;
      const bool in = i < n1 && j < n2;
      q[h][u] = in ? in_q[i * n2 + j] : 0.f;
      t[h][u] = in && in_t ? in_t[i * n2 + j] : 0.f;
    }
  for (int l = 0; l < run.n; ++l) {
    const ntg_flat_layer_t& ly = run.layer[l];
    if (ly.has_affine) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float a, b = 0.f;
          apply_affine(ly.aff, q[h][u], t[h][u], out_t != nullptr, a, b);
          q[h][u] = a;
          t[h][u] = b;
        }
    }
    if (ly.act.kind != NTG_ACT_NONE) {
      const ActC ac = act_consts(ly.act);
      const float* v = fv + (2 * l) * kFlatSamples;
      const float* s = v + kFlatSamples;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float v2 = v[kFlatRows + lane + 32 * h], sv2 = s[kFlatRows + lane + 32 * h];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          act_apply<!RELU, !RELU>(ac, q[h][u], t[h][u], v[w + u], v2, s[w + u], sv2);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = r0 + w + u, j = c0 + lane + 32 * h;
      if (i >= n1 || j >= n2) continue;
      out_q[i * n2 + j] = q[h][u];
      if (out_t) out_t[i * n2 + j] = t[h][u];
    }
}

bool rows_vec(const float* x1, const float* x2, int64_t d) {
  return (d & 3) == 0 &&
         ((reinterpret_cast<uintptr_t>(x1) | reinterpret_cast<uintptr_t>(x2)) & 15) == 0;
}

template <int T, int BK, int RU, int RV>
void launch_gram_small(bool sym, bool vec, cudaStream_t s, const float* x1, const float* x2,
                       int64_t n1, int64_t n2, int64_t d, float* out) {
  const int64_t nb1 = ceil_div(n1, T), nb2 = ceil_div(n2, T);
  const float inv = 1.f / (float)d;
  const dim3 block(16 * (T / RU));
  if (sym) {
    const dim3 grid((unsigned)(nb1 * (nb1 + 1) / 2));
    if (vec) gram_small_kernel<T, BK, RU, RV, true, true><<<grid, block, 0, s>>>(x1, x2, n1, n2, d, inv, out);
    else gram_small_kernel<T, BK, RU, RV, true, false><<<grid, block, 0, s>>>(x1, x2, n1, n2, d, inv, out);
  } else {
    const dim3 grid((unsigned)nb2, (unsigned)nb1);
    if (vec) gram_small_kernel<T, BK, RU, RV, false, true><<<grid, block, 0, s>>>(x1, x2, n1, n2, d, inv, out);
    else gram_small_kernel<T, BK, RU, RV, false, false><<<grid, block, 0, s>>>(x1, x2, n1, n2, d, inv, out);
  }
}

}  // namespace

namespace {

// Small products C[M, N] (+)= alpha op(A) B, op(A) = A [M, K] or (TA) A^T with A [K, M]: 32 x 32
// tiles, 2 x 2 outputs per thread, slices of 16 streamed by a 4-stage cp.async ring. Bound by
// the chain of K / 16 slices, so the sums can afford to be better than one long chain: each
// slice is summed by itself and added with its rounding error kept (two-sum).
template <bool TA>
__global__ void __launch_bounds__(256)
    gemm_small_kernel(const float* __restrict__ A, const float* __restrict__ B,
                      float* __restrict__ C, int64_t M, int64_t N, int64_t K, float alpha,
                      int accumulate) {
  constexpr int T = 32, BK = 16, ST = 4, PA = TA ? T + 4 : BK + 4, RA = TA ? BK : T;
  __shared__ __align__(16) float As[ST][RA * PA];
  __shared__ __align__(16) float Bs[ST][BK * (T + 4)];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t row0 = (int64_t)blockIdx.y * T, col0 = (int64_t)blockIdx.x * T;
  const int64_t nk = (K + BK - 1) / BK;
  auto stage = [&](int64_t s) {
    if (s < nk) {
      // rows of A (of length K, or M when transposed) and of B (length N), 4 bytes a copy
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int idx = threadIdx.x + 256 * e;
        if (TA) {
          const int r = idx >> 5, c = idx & 31;
          const int64_t gk = s * BK + r, gi = row0 + c;
          const bool in = gk < K && gi < M;
          cp_async<false>(&As[s % ST][r * PA + c], in ? A + gk * M + gi : A, in);
        } else {
          const int r = idx >> 4, c = idx & 15;
          const int64_t gk = s * BK + c, gi = row0 + r;
          const bool in = gk < K && gi < M;
          cp_async<false>(&As[s % ST][r * PA + c], in ? A + gi * K + gk : A, in);
        }
        const int r = idx >> 5, c = idx & 31;
        const int64_t gk = s * BK + r, gj = col0 + c;
        const bool in = gk < K && gj < N;
        cp_async<false>(&Bs[s % ST][r * (T + 4) + c], in ? B + gk * N + gj : B, in);
      }
    }
    cp_commit();
  };
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) stage(s);
  float hi[2][2] = {}, lo[2][2] = {};
  for (int64_t s = 0; s < nk; ++s) {
    cp_wait<ST - 2>();
    __syncthreads();
    stage(s + ST - 1);
    const float* a = As[s % ST];
    const float* b = Bs[s % ST];
    float p[2][2] = {};
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float2 bv = *reinterpret_cast<const float2*>(b + k * (T + 4) + 2 * tx);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float av = TA ? a[k * PA + 2 * ty + u] : a[(2 * ty + u) * PA + k];
        p[u][0] = fmaf(av, bv.x, p[u][0]);
        p[u][1] = fmaf(av, bv.y, p[u][1]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const float t = __fadd_rn(hi[u][v], p[u][v]);
        const float z = __fsub_rn(t, hi[u][v]);
        lo[u][v] += __fadd_rn(__fsub_rn(hi[u][v], __fsub_rn(t, z)), __fsub_rn(p[u][v], z));
        hi[u][v] = t;
      }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int64_t gi = row0 + 2 * ty + u, gj = col0 + 2 * tx + v;
      if (gi >= M || gj >= N) continue;
      float* c = C + gi * N + gj;
      // an infinite or NaN sum has no rounding error to add
      const float r = alpha * (isfinite(hi[u][v]) ? hi[u][v] + lo[u][v] : hi[u][v]);
      *c = accumulate ? *c + r : r;
    }
}

}  // namespace

bool gemm_small(cudaStream_t s, const float* a, const float* b, float* c, int64_t m, int64_t n,
                int64_t k, bool trans_a, float alpha, bool accumulate) {
  // below one 64 x 64 tile per SM: the eigenvectors of 500 points times 60 columns take 16 us
  // (57 us on eight 64 x 64 tiles); whole calls on 64 x 64 tiles and here, plain and with A
  // transposed: 200^3 38, 48 and 28, 27 us, 500^3 64, 85 and 43, 44, 640^3 77, 104 and 61, 62,
  // 768^3 (144 tiles) 86, 121 and 81, 82, 768 x 768 x 4096 368, 554 and 334, 347
  if (ceil_div(m, 64) * ceil_div(n, 64) >= 152 || ceil_div(m, 32) > 65535) return false;
  const dim3 grid((unsigned)ceil_div(n, 32), (unsigned)ceil_div(m, 32));
  if (trans_a)
    gemm_small_kernel<true><<<grid, 256, 0, s>>>(a, b, c, m, n, k, alpha, accumulate);
  else
    gemm_small_kernel<false><<<grid, 256, 0, s>>>(a, b, c, m, n, k, alpha, accumulate);
  return true;
}

int gram_fp32(cudaStream_t s, const float* x1, const float* x2, int64_t n1, int64_t n2, int64_t d,
              float* out) {
  NTG_REQUIRE(ceil_div(n1, 128) <= 65535, "ntg_gram: n1 too large");
  const bool sym = x1 == x2 && n1 == n2;  // the lower triangle of tiles, mirrored
  const bool vec = rows_vec(x1, x2, d);
  auto tiles = [&](int64_t t) {
    const int64_t a = ceil_div(n1, t), b = ceil_div(n2, t);
    return sym ? a * (a + 1) / 2 : a * b;
  };
  // The largest tile that still gives every SM one: a tile costs the same whatever else
  // runs, and a smaller one reads more of its operands per output. Calls on 128-wide tiles and
  // on the ones taken here: 300^2 x 784 120 and 32 us, 700^2 121 and 53 (32 wide), 1000^2 121 and
  // 73, 1200 x 1100 x 3072 417 and 305 (64 wide); at 1500^2 (144 tiles of 128) 122 and 120.
  if (tiles(128) >= 152) {
    const float inv = 1.f / (float)d;
    const int64_t nb1 = ceil_div(n1, 128);
    const dim3 grid = sym ? dim3((unsigned)tiles(128)) : dim3((unsigned)ceil_div(n2, 128), (unsigned)nb1);
    if (sym && vec) gram_simt_kernel<true, true><<<grid, 256, 0, s>>>(x1, x2, n1, n2, d, inv, out);
    else if (sym) gram_simt_kernel<true, false><<<grid, 256, 0, s>>>(x1, x2, n1, n2, d, inv, out);
    else if (vec) gram_simt_kernel<false, true><<<grid, 256, 0, s>>>(x1, x2, n1, n2, d, inv, out);
    else gram_simt_kernel<false, false><<<grid, 256, 0, s>>>(x1, x2, n1, n2, d, inv, out);
  } else if (tiles(64) >= 152) {
    launch_gram_small<64, 16, 4, 4>(sym, vec, s, x1, x2, n1, n2, d, out);
  } else {
    launch_gram_small<32, 32, 4, 2>(sym, vec, s, x1, x2, n1, n2, d, out);
  }
  note_launch();
  return check_launch("ntg_gram");
}

int cov_rows(cudaStream_t s, const float* x1, int64_t n1, const float* x2, int64_t n2, int64_t d,
             float* cov1, float* cov2) {
  const unsigned grid = (unsigned)(ceil_div(n1, 32) + ceil_div(n2, 32));
  const float inv = 1.f / (float)d;
  if (rows_vec(x1, n2 > 0 ? x2 : x1, d))
    cov_diag_kernel<true><<<grid, 128, 0, s>>>(x1, n1, x2, n2, d, inv, cov1, cov2);
  else
    cov_diag_kernel<false><<<grid, 128, 0, s>>>(x1, n1, x2, n2, d, inv, cov1, cov2);
  note_launch();
  return check_launch("ntg_cov_diag");
}

}  // namespace ntg

using namespace ntg;

extern "C" size_t ntg_gram_workspace_bytes(int64_t n1, int64_t n2, int64_t d) {
  return gram_tc_workspace(n1, n2, d);
}

extern "C" int ntg_gram(void* stream, const float* x1, const float* x2, int64_t n1, int64_t n2,
                        int64_t d, float* nngp, int32_t precision, void* workspace,
                        size_t workspace_bytes) {
  NTG_REQUIRE(x1 && x2 && nngp, "ntg_gram: null pointer");
  NTG_REQUIRE(n1 > 0 && n2 > 0 && d > 0, "ntg_gram: sizes must be positive");
  if (precision == 1) {
    return gram_tc(as_stream(stream), x1, x2, n1, n2, d, nngp, workspace, workspace_bytes);
  }
  NTG_REQUIRE(precision == 0, "ntg_gram: precision must be 0 or 1");
  return gram_fp32(as_stream(stream), x1, x2, n1, n2, d, nngp);
}

extern "C" int ntg_cov_diag(void* stream, const float* x, int64_t n, int64_t d, float* cov) {
  NTG_REQUIRE(x && cov, "ntg_cov_diag: null pointer");
  NTG_REQUIRE(n > 0 && d > 0, "ntg_cov_diag: sizes must be positive");
  return cov_rows(as_stream(stream), x, n, nullptr, 0, d, cov, nullptr);
}

extern "C" int ntg_flat_rules(void* stream, const float* in_q, const float* in_t, int64_t n1,
                              int64_t n2, const float* var1, int64_t s1, const float* var2,
                              int64_t s2, int32_t n_layers, const ntg_flat_layer_t* layers,
                              float* out_q, float* out_t, float* cov1, float* cov2) {
  NTG_REQUIRE(in_q && var1 && var2 && layers && out_q, "ntg_flat_rules: null pointer");
  NTG_REQUIRE(n1 > 0 && n2 > 0 && s1 > 0 && s2 > 0, "ntg_flat_rules: bad sizes");
  NTG_REQUIRE(n_layers > 0 && n_layers <= NTG_FLAT_MAX_LAYERS, "ntg_flat_rules: bad layer count");
  FlatRun run;
  run.n = n_layers;
  bool relu = true;
  for (int l = 0; l < n_layers; ++l) {
    const ntg_act_t& a = layers[l].act;
    NTG_REQUIRE(a.kind >= NTG_ACT_NONE && a.kind <= NTG_ACT_GELU,
                "ntg_flat_rules: unknown activation kind");
    relu = relu && (a.kind == NTG_ACT_NONE || (a.kind == NTG_ACT_ABRELU && a.stabilize <= 0.f));
    run.layer[l] = layers[l];
  }
  const int64_t blocks = ceil_div(n1, kFlatRows) * ceil_div(n2, kFlatCols);
  NTG_REQUIRE(blocks < (1ll << 31), "ntg_flat_rules: kernel too large");
  const size_t sm = sizeof(float) * 2 * kFlatSamples * n_layers;
  cudaStream_t s = as_stream(stream);
  if (relu)
    flat_rules_kernel<true><<<(unsigned)blocks, 256, sm, s>>>(run, in_q, in_t, n1, n2, var1, s1,
                                                              var2, s2, out_q, out_t, cov1, cov2);
  else
    flat_rules_kernel<false><<<(unsigned)blocks, 256, sm, s>>>(run, in_q, in_t, n1, n2, var1, s1,
                                                               var2, s2, out_q, out_t, cov1, cov2);
  note_launch();
  return check_launch("ntg_flat_rules");
}

extern "C" int ntg_flat_input(void* stream, const float* x1, const float* x2, int64_t n1,
                              int64_t n2, int64_t d, float* nngp, float* cov1, float* cov2,
                              int32_t precision, void* workspace, size_t workspace_bytes) {
  const int rc = ntg_gram(stream, x1, x2, n1, n2, d, nngp, precision, workspace, workspace_bytes);
  if (rc != NTG_OK || !cov1) return rc;
  NTG_REQUIRE(cov2, "ntg_flat_input: cov1 and cov2 go together");
  return cov_rows(as_stream(stream), x1, n1, x2, n2, d, cov1, cov2);
}
