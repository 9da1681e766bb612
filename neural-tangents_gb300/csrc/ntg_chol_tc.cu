// Blocked Cholesky factorisation and solves of predict.gradient_descent_mse on
// the sm_103a tensor cores (neural_tangents/_src/predict.py:1224-1258 restated
// for the GPU): A = K + lambda I = L L^T in FP32 with 128-wide panels.
//
// Per panel k, on a chain of its own:
//   diag_block_kernel   one CTA factors the 128 x 128 diagonal block (four
//                       32-wide steps, each a warp-level Cholesky + inverse in
//                       registers overlapped with the other warps' deferred
//                       updates, then the sub-panel and the next column block as
//                       register-tiled warp products in shared memory) and writes
//                       the block's inverse L11^-1;
//   next_tile_kernel    the first tile of the rows below, L21 = A21 L11^-T as a product with
//                       that inverse, and its update of the next diagonal block;
// beside it:
//   gemm_tf32x3         the other rows of L21 (in place, one 128-wide column of tiles) and
//                       of the next column block;
//   gemm_tf32x3 lower   the trailing update A22 -= L21 L21^T on the tensor cores
//                       (3xTF32 products, FP32 accumulation; tiles on or below the
//                       diagonal only).
// After the panels, the explicit inverse factors L^-T (a forward block solve of
// L Y = I on the tensor cores, only the non-zero rows of each block column) and
// L^-1 (its transpose) are kept in the factor workspace: a solve is then two
// triangular products, GEMV-shaped for up to kSmallM right-hand sides (a warp
// per row, bandwidth-bound) and tensor-core GEMMs for more.
// Refinement keeps x in FP64 and accumulates every product with K in
// double-float (two FP32 words, error-free products and sums; about 44
// significant bits), which the GB300's FP32 rate makes about 6x cheaper than
// FP64: for up to kSmallM right-hand sides preconditioned conjugate gradients
// (the factor as preconditioner; converges where plain refinement stalls,
// kappa u > 1, each column stopping once its residual fell by kPcgTol), for
// more, refine_iters steps of x <- x + (L L^T)^-1 (b - A x).
#include <mutex>
#include <string>

#include "ntg_common.cuh"
#include "ntg_exact_tc.cuh"

namespace ntg {
int gemm_tf32x3(cudaStream_t s, const float* a, int64_t lda, const float* b, int64_t ldb,
                float* c, int64_t ldc, int64_t m, int64_t n, int64_t k, float alpha, float beta,
                int lower, int tri = 0);

namespace {

constexpr int PB = 128;        // panel / diagonal block
constexpr int PBS = PB + 1;    // padded shared-memory row
constexpr int XP = PB + 4;     // pitch of the p-major / 16-byte-row shared-memory tiles
constexpr int kSmallM = 16;    // right-hand sides of the cooperative solves
constexpr int kGT = 128;       // rows of a split-K product tile (one per thread)
constexpr int kGK = 32;        // columns staged in shared memory per step

__host__ __device__ __forceinline__ int64_t mini(int64_t a, int64_t b) { return a < b ? a : b; }

// Grid of a grid-stride loop over n elements, 256 threads a block.
int grid_for(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g > 152 * 32 ? 152 * 32 : (g < 1 ? 1 : g));
}

// ---------------------------------------------------------------------------
// Set-up
// ---------------------------------------------------------------------------

__global__ void trace_tc_kernel(const float* __restrict__ A, int64_t n, double* __restrict__ out) {
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += (double)A[i * n + i];
  __shared__ double part[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    out[0] = t;
  }
}

// L[i, j] = A[i, j] (j < i), A[i, i] + lambda (j == i), 0 above the diagonal and in the
// padding columns n <= j < ldl; Z = I, padded alike. A row per blockIdx.y: bound by the two arrays that it writes (n 5000: 41 us; two kernels over entries
// 96).
__global__ void __launch_bounds__(256)
    init_factor_ld_kernel(const float* __restrict__ A, int64_t n, int64_t ldl, double reg,
                          int absolute, const double* __restrict__ trace, float* __restrict__ L,
                          float* __restrict__ Z, double* __restrict__ lambda) {
  // FP64 is slow here: a division by every thread takes longer than the kernel
  auto lam = [&] { return absolute ? reg : reg * trace[0] / (double)n; };
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) lambda[0] = lam();
  const int64_t i = blockIdx.y, j0 = (int64_t)blockIdx.x * 1024 + threadIdx.x;
  const float* a = A + i * n;
  float v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int64_t j = j0 + 256 * u;
    v[u] = j <= i ? __ldg(a + j) : 0.f;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int64_t j = j0 + 256 * u;
    if (j >= ldl) break;
    L[i * ldl + j] = v[u];
    Z[i * ldl + j] = j == i ? 1.f : 0.f;
    if (j == i) L[i * ldl + j] = (float)((double)v[u] + lam());
  }
}

// ---------------------------------------------------------------------------
// What the next diagonal block waits for
// ---------------------------------------------------------------------------

// d += A B^T of one m16n8k8 TF32 product (mma.sync, row-major A, B given as rows of k).
__device__ __forceinline__ void mma_tf32_16x8(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                              uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}

// The first tile of panel k, L21 = A21 L11^-T (UPDATE false: rows k + 128 .., in place), then its
// update of the diagonal block behind it, A22 -= L21 L21^T (UPDATE, lower part): all that the
// next diagonal block waits for. Eight CTAs of 16 rows, each warp 16 columns, 3xTF32 on
// mma.sync straight from L2: 128 x 128 x 128 is too short for the set-up of a tcgen05 pipeline
// (10 - 13 us and a gap of 3 - 5 in gemm_tf32x3, 5 us here with the launches overlapped; both
// products in one CTA 27 us), and without shared memory the CTAs fit beside those of the
// trailing update. A panel of a 5000-point factorisation takes 50 - 58 us (66), bound from
// there on by the trailing update and the inverse, which share the SMs.
template <bool UPDATE>
__global__ void __launch_bounds__(256)
    next_tile_kernel(float* __restrict__ L, int64_t ldl, int64_t n, int64_t k, const float* linv) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nb = (int)mini(PB, n - k - PB);
  const int r0 = blockIdx.x * 16, c0 = (threadIdx.x >> 5) * 16;
  float* const a21 = L + (k + PB) * ldl + k;
  const bool idle = UPDATE && c0 > r0 + 15;
  // L11^-1 is lower triangular: its rows c0 .. c0 + 15 end at column c0 + 15
  const int K = UPDATE ? PB : c0 + 16;
  const float* const B = UPDATE ? a21 : linv;
  const int64_t ldb = UPDATE ? ldl : PB;
  const int nbr = UPDATE ? nb : PB;
  after_previous();
  if (idle) return;
  float acc[2][4] = {};
  // Thread t of four holds the words 4 t .. 4 t + 3 of 16 consecutive k and hands them to two
  // products, (0, 1) as their k = t and t + 4, then (2, 3): the same order of k in A and B.
#pragma unroll 4
  for (int kb = 0; kb < K; kb += 16) {
    float4 av[2], bv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int ra = r0 + g + 8 * h, rb = c0 + g + 8 * h;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      av[h] = ra < nb ? *reinterpret_cast<const float4*>(a21 + ra * ldl + kb + 4 * t) : zero;
      bv[h] = rb < nbr ? *reinterpret_cast<const float4*>(B + rb * ldb + kb + 4 * t) : zero;
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      uint32_t ah[4], al[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        split_tf32(s ? av[h].z : av[h].x, ah[h], al[h]);
        split_tf32(s ? av[h].w : av[h].y, ah[2 + h], al[2 + h]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t h0, l0, h1, l1;
        split_tf32(s ? bv[j].z : bv[j].x, h0, l0);
        split_tf32(s ? bv[j].w : bv[j].y, h1, l1);
        mma_tf32_16x8(acc[j], al, h0, h1);
        mma_tf32_16x8(acc[j], ah, l0, l1);
        mma_tf32_16x8(acc[j], ah, h0, h1);
      }
    }
  }
  if (!UPDATE) __syncthreads();  // the rows are read by every warp before they are written
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = r0 + g + 8 * (e >> 1), c = c0 + 8 * j + 2 * t + (e & 1);
      if (i >= nb) continue;
      if (!UPDATE) a21[i * ldl + c] = acc[j][e];
      else if (c <= i) a21[i * ldl + PB + c] -= acc[j][e];
    }
}

// ---------------------------------------------------------------------------
// Diagonal block: factor + inverse (one CTA of 512 threads)
// ---------------------------------------------------------------------------

// Warp-level Cholesky of the 32 x 32 block at (o, o) of `a` and the inverse of the
// factor. Lane r holds row r in registers; each pivot is broadcast by a shuffle and each
// finished column of L is stored to lt[j][:] (zeros above the diagonal), from where the
// rank-1 update and the inverse read it as broadcast 16-byte words. The pivot uses the
// hardware reciprocal square root (2 ulp): L_jj = d rsqrt(d), L_rj = A_rj rsqrt(d); the
// reciprocal pivots are kept for the inverse, which then needs no division (the factor
// is refined against the exact kernel by the solves). Lane c computes column c of
// X = L^-1 column-sweep style (x_p = s_p / L_pp, then s_i -= L_ip x_p for every i > p),
// so the updates of a step are independent. Writes the factor into a (upper part zero)
// and X row-major into dinv (pitch 33) and into xs at (o, o) (pitch XP).
__device__ void warp_potrf_inv32(float (*a)[PBS], int o, float (*dinv)[33], float* xs,
                                 int* info, int64_t col0) {
  __shared__ __align__(16) float lt[32][36];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float v[32], rp[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = a[o + lane][o + c];
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float d = __shfl_sync(full, v[j], j);
    if (!(d > 0.f)) {  // the same value in every lane
      if (lane == 0) atomicCAS(info, 0, (int)(col0 + o + j + 1));
      d = 1.f;
    }
    const float rs = rsqrtf(d);
    rp[j] = rs;
    const float l = (lane == j) ? d * rs : v[j] * rs;  // lanes < j: the unused upper part
    v[j] = l;
    lt[j][lane] = lane >= j ? l : 0.f;
    __syncwarp();
#pragma unroll
    for (int q = (j + 1) / 4; q < 8; ++q) {
      const float4 c4 = *reinterpret_cast<const float4*>(&lt[j][4 * q]);
      const float cv[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (4 * q + u > j) v[4 * q + u] = fmaf(-l, cv[u], v[4 * q + u]);
    }
  }
#pragma unroll
  for (int c = 0; c < 32; ++c) a[o + lane][o + c] = (c <= lane) ? v[c] : 0.f;
  float x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = (i == lane) ? 1.f : 0.f;
#pragma unroll
  for (int p = 0; p < 32; ++p) {
    const float xp = x[p] * rp[p];
    x[p] = xp;
#pragma unroll
    for (int q = (p + 1) / 4; q < 8; ++q) {
      const float4 c4 = *reinterpret_cast<const float4*>(&lt[p][4 * q]);
      const float cv[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (4 * q + u > p) x[4 * q + u] = fmaf(-cv[u], xp, x[4 * q + u]);
    }
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    dinv[i][lane] = x[i];
    xs[(o + i) * XP + o + lane] = x[i];
  }
  __syncwarp();
}

// acc[i][j] += sum_{p < 32} A(r0 + i, p) B(p, c0 + j) for the 8 x 4 piece of a 32 x 32
// tile that lane (r0 / 8) * 8 + c0 / 4 owns. AP: A is p-major (A[p * lda + r], two
// 16-byte loads per p), else row-major (A[r * lda + p]); BP: B is p-major (B[p * ldb + c],
// one 16-byte load), else transposed (B[c * ldb + p]). Row-major pitches 129 / 33 and
// p-major pitch XP keep the loads of a warp free of bank conflicts.
template <bool AP, bool BP>
__device__ __forceinline__ void warp_tile_acc(float (&acc)[8][4], const float* A, int lda,
                                              const float* B, int ldb) {
  const int lane = threadIdx.x & 31;
  const int r0 = (lane >> 3) * 8, c0 = (lane & 7) * 4;
#pragma unroll 4
  for (int p = 0; p < 32; ++p) {
    float av[8], bv[4];
    if (AP) {
      const float4 x = *reinterpret_cast<const float4*>(A + p * lda + r0);
      const float4 y = *reinterpret_cast<const float4*>(A + p * lda + r0 + 4);
      av[0] = x.x; av[1] = x.y; av[2] = x.z; av[3] = x.w;
      av[4] = y.x; av[5] = y.y; av[6] = y.z; av[7] = y.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = A[(r0 + i) * lda + p];
    }
    if (BP) {
      const float4 z = *reinterpret_cast<const float4*>(B + p * ldb + c0);
      bv[0] = z.x; bv[1] = z.y; bv[2] = z.z; bv[3] = z.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = B[(c0 + j) * ldb + p];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
}

__device__ __forceinline__ void zero_acc(float (&acc)[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
}

// a[32 I + r][32 J + c] -= sum_p P[32 I + r][p] P[32 J + c][p], P the panel held
// p-major in pt (one warp, one 32 x 32 tile).
__device__ __forceinline__ void warp_update_tile(float (*a)[PBS], const float* pt, int I, int J) {
  const int lane = threadIdx.x & 31;
  const int r0 = (lane >> 3) * 8, c0 = (lane & 7) * 4;
  float acc[8][4];
  zero_acc(acc);
  warp_tile_acc<true, true>(acc, pt + 32 * I, XP, pt + 32 * J, XP);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a[32 * I + r0 + i][32 * J + c0 + j] -= acc[i][j];
}

// Factors L[k:k+nb, k:k+nb] in place (upper part zeroed) and writes the inverse of the
// factor, zero-padded to 128 x 128, to linv (row-major). Four 32-wide steps; in step sb:
//   phase A  warp 0 factors and inverts diagonal block sb (warp_potrf_inv32) while the
//            other warps apply the previous panel's update to the column blocks beyond
//            sb + 1 (deferred: only block sb + 1 must be current for the next step) and
//            form T_j = sum_{q=j}^{sb-1} L_{sb,q} X_{q,j}, j < sb, for the inverse;
//   phase B  X_{sb,j} = -Dinv_sb T_j, and the sub-panel L_{rb,sb} = A_{rb,sb} Dinv_sb^T
//            for the row blocks rb > sb (into a and, p-major, into pt);
//   phase C  the update of column block sb + 1 by panel sb.
// Every product is a 32 x 32 x 32 warp tile (warp_tile_acc). Rows beyond nb are
// padded with the identity (which factors and inverts to itself and is cut on output).
__global__ void __launch_bounds__(512, 1)
    diag_block_kernel(float* __restrict__ L, int64_t ldl, int64_t n, int64_t k, int* info,
                      float* __restrict__ linv) {
  extern __shared__ __align__(16) float sm[];
  float(*a)[PBS] = reinterpret_cast<float(*)[PBS]>(sm);  // 128 x 129, the block
  float* pt = sm + PB * PBS;                              // 32 x XP, current panel p-major
  float* xs = pt + 32 * XP;                               // 128 x XP, X = L^-1
  float* tb = xs + PB * XP;                               // 32 x XP, T_j at columns 32 j
  float(*dinv)[32][33] = reinterpret_cast<float(*)[32][33]>(tb + 32 * XP);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = (lane >> 3) * 8, c0 = (lane & 7) * 4;
  const int nb = (int)mini(PB, n - k);
  after_previous();
  if (nb == PB) {
    // full block (16-byte aligned: ldl % 4 == 0, k % 128 == 0): all eight 16-byte loads
    // of a thread in flight at once; entries above the diagonal are not read
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = tid + 512 * u, i = e >> 5, j = (e & 31) * 4;
      v[u] = j <= i ? *reinterpret_cast<const float4*>(L + (k + i) * ldl + k + j)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = tid + 512 * u, i = e >> 5, j = (e & 31) * 4;
      a[i][j] = v[u].x;
      a[i][j + 1] = j + 1 <= i ? v[u].y : 0.f;
      a[i][j + 2] = j + 2 <= i ? v[u].z : 0.f;
      a[i][j + 3] = j + 3 <= i ? v[u].w : 0.f;
    }
  } else {
    for (int idx = tid; idx < PB * PB; idx += 512) {
      const int i = idx >> 7, j = idx & (PB - 1);
      float v;
      if (i < nb && j < nb) v = (j <= i) ? L[(k + i) * ldl + k + j] : 0.f;
      else v = (i == j) ? 1.f : 0.f;
      a[i][j] = v;
    }
  }
  __syncthreads();
  for (int sb = 0; sb < 4; ++sb) {
    const int o = 32 * sb;
    // ---- phase A ----
    if (warp == 0) {
      warp_potrf_inv32(a, o, dinv[sb], xs, info, k);
    } else if (sb > 0) {
      const int u = warp - 1;
      int cnt = 0;
      for (int J = sb + 1; J < 4; ++J)
        for (int I = J; I < 4; ++I, ++cnt)
          if (cnt == u) warp_update_tile(a, pt, I, J);
      for (int j = 0; j < sb; ++j, ++cnt) {
        if (cnt != u) continue;
        float acc[8][4];
        zero_acc(acc);
        for (int q = j; q < sb; ++q)
          warp_tile_acc<false, true>(acc, &a[o][32 * q], PBS, xs + 32 * q * XP + 32 * j, XP);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4*>(tb + (r0 + i) * XP + 32 * j + c0) =
              make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      }
    }
    __syncthreads();
    // ---- phase B ----
    {
      const int u = warp;
      if (u < sb) {  // X_{sb,u} = -Dinv_sb T_u
        float acc[8][4];
        zero_acc(acc);
        warp_tile_acc<false, true>(acc, &dinv[sb][0][0], 33, tb + 32 * u, XP);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4*>(xs + (o + r0 + i) * XP + 32 * u + c0) =
              make_float4(-acc[i][0], -acc[i][1], -acc[i][2], -acc[i][3]);
      } else if (u < 3) {  // sub-panel row block rb = sb + 1 + (u - sb)
        const int rb = u + 1;
        if (rb > sb) {
          float acc[8][4];
          zero_acc(acc);
          warp_tile_acc<false, false>(acc, &a[32 * rb][o], PBS, &dinv[sb][0][0], 33);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) a[32 * rb + r0 + i][o + c0 + j] = acc[i][j];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float* d = pt + (c0 + j) * XP + 32 * rb + r0;
            *reinterpret_cast<float4*>(d) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            *reinterpret_cast<float4*>(d + 4) =
                make_float4(acc[4][j], acc[5][j], acc[6][j], acc[7][j]);
          }
        }
      }
    }
    __syncthreads();
    // ---- phase C ----
    if (sb < 3) {
      const int I = sb + 1 + warp;
      if (I < 4) warp_update_tile(a, pt, I, sb + 1);
      __syncthreads();
    }
  }
  // the factor (lower incl. the diagonal; upper zero) and the inverse
  if (nb == PB) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = tid + 512 * u, i = e >> 5, j = (e & 31) * 4;
      const float4 lv = make_float4(a[i][j], j + 1 <= i ? a[i][j + 1] : 0.f,
                                    j + 2 <= i ? a[i][j + 2] : 0.f,
                                    j + 3 <= i ? a[i][j + 3] : 0.f);
      *reinterpret_cast<float4*>(L + (k + i) * ldl + k + j) =
          j <= i ? lv : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xv = (j >> 5) <= (i >> 5) ? *reinterpret_cast<const float4*>(xs + i * XP + j)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(linv + i * PB + j) = xv;
    }
  } else {
    for (int idx = tid; idx < nb * nb; idx += 512) {
      const int i = idx / nb, j = idx - i * nb;
      L[(k + i) * ldl + k + j] = (j <= i) ? a[i][j] : 0.f;
    }
    for (int idx = tid; idx < PB * PB; idx += 512) {
      const int i = idx >> 7, j = idx & (PB - 1);
      const bool in = i < nb && j < nb && (j >> 5) <= (i >> 5);
      linv[idx] = in ? xs[i * XP + j] : 0.f;
    }
  }
}

constexpr size_t kDiagSmem = (size_t)(PB * PBS + 32 * XP + PB * XP + 32 * XP + 4 * 32 * 33) *
                             sizeof(float);

// out[j, i] = in[i, j] for an [rows, cols] block (row pitches ld_in, ld_out); upper: in is zero
// below its diagonal, and the tiles there are not read (n 5000: 36 us instead of 63).
__global__ void __launch_bounds__(256)
    transpose_kernel(const float* __restrict__ in, int64_t ld_in, float* __restrict__ out,
                     int64_t ld_out, int64_t rows, int64_t cols, bool upper) {
  __shared__ float tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, c0 = (int64_t)blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const bool zero = upper && c0 + 31 < r0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = ty + 8 * u;
    const int64_t r = r0 + i, c = c0 + tx;
    tile[i][tx] = (r < rows && c < cols && !zero) ? in[r * ld_in + c] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = ty + 8 * u;
    const int64_t c = c0 + i, r = r0 + tx;
    if (c < cols && r < rows) out[c * ld_out + r] = tile[tx][i];
  }
}

// ---------------------------------------------------------------------------
// Residuals R = B - (A + lambda I) X with X in FP64.
// ---------------------------------------------------------------------------

__global__ void max_abs64_kernel(const double* __restrict__ v, int64_t n, double* __restrict__ out) {
  double mx = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    mx = fmax(mx, fabs(v[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(out),
              (unsigned long long)__double_as_longlong(mx));
}


__device__ __forceinline__ P2 neg2(P2 x) {
  P2 r;
  asm("xor.b64 %0, %1, 0x8000000080000000;" : "=l"(r.v) : "l"(x.v));
  return r;
}

// Double-float multiply-add on two lanes at once: (sh, sl) += a (xh + xl) with a FP32 and
// (xh, xl), (sh, sl) double-float pairs: the product a xh split exactly into ph + pl by a
// fused multiply-add, a xl added to pl, ph added to sh by the error-free two-sum (its
// rounding error to the low word), as in the accurate dot products of Ogita, Rump and
// Oishi (2005).
__device__ __forceinline__ void df_fma2(P2 a, P2 xh, P2 xl, P2& sh, P2& sl) {
  const P2 ph = mul2(a, xh);
  P2 pl = fma2(a, xh, neg2(ph));
  pl = fma2(a, xl, pl);
  const P2 sum = add2(sh, ph);
  const P2 bv = sub2(sum, sh);
  const P2 e = add2(sub2(sh, sub2(sum, bv)), sub2(ph, bv));
  sl = add2(sl, add2(e, pl));
  sh = sum;
}

// Double-float residual over 64 x 64 tiles of (row, column): R = B - (A + lambda I) X
// (B64 in place of B when given),
// the products taken with X's double-float split xs (split_df_kernel: split once, not
// once per tile). Each thread keeps 4 x 4 sums as 4 x 2 packed pairs of columns
// (df_fma2); rnorm receives max |R|.
__global__ void __launch_bounds__(256)
    residual_df_kernel(const float* __restrict__ A, int64_t n, const double* lambda,
                       const float* __restrict__ B, const double* __restrict__ B64,
                       const double* __restrict__ X,
                       const float2* __restrict__ xs, int64_t m, float* __restrict__ R,
                       double* __restrict__ rnorm) {
  __shared__ float As[16][64 + 1];   // [k][i]
  __shared__ float Xh[16][64 + 1];   // [k][j]
  __shared__ float Xl[16][64 + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t i0 = (int64_t)blockIdx.y * 64, j0 = (int64_t)blockIdx.x * 64;
  P2 sh[4][2], sl[4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) sh[u][v] = sl[u][v] = p2s(0.f);
  for (int64_t k0 = 0; k0 < n; k0 += 16) {
    for (int idx = threadIdx.x; idx < 16 * 64; idx += 256) {
      const int i = idx / 16, k = idx % 16;
      As[k][i] = (i0 + i < n && k0 + k < n) ? A[(i0 + i) * n + k0 + k] : 0.f;
      const int kk = idx / 64, j = idx % 64;
      const float2 xv = (k0 + kk < n && j0 + j < m) ? xs[(k0 + kk) * m + j0 + j]
                                                    : make_float2(0.f, 0.f);
      Xh[kk][j] = xv.x;
      Xl[kk][j] = xv.y;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      P2 av[4], hv[2], lv[2];
#pragma unroll
      for (int u = 0; u < 4; ++u) av[u] = p2s(As[k][ty * 4 + u]);
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        hv[v] = p2(Xh[k][tx * 4 + 2 * v], Xh[k][tx * 4 + 2 * v + 1]);
        lv[v] = p2(Xl[k][tx * 4 + 2 * v], Xl[k][tx * 4 + 2 * v + 1]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) df_fma2(av[u], hv[v], lv[v], sh[u][v], sl[u][v]);
    }
    __syncthreads();
  }
  double rmax = 0.0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int64_t i = i0 + ty * 4 + u;
    if (i >= n) continue;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int64_t j = j0 + tx * 4 + v;
      if (j >= m) continue;
      float h0, h1, l0, l1;
      p2u(sh[u][v >> 1], h0, h1);
      p2u(sl[u][v >> 1], l0, l1);
      const double ax = (v & 1) ? (double)h1 + (double)l1 : (double)h0 + (double)l0;
      const double b = B64 ? B64[i * m + j] : (double)B[i * m + j];
      const double r = b - ax - lambda[0] * X[i * m + j];
      R[i * m + j] = (float)r;
      rmax = fmax(rmax, fabs(r));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
  if ((threadIdx.x & 31) == 0 && rmax > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(rnorm),
              (unsigned long long)__double_as_longlong(rmax));
}

__global__ void to_double_tc_kernel(const float* __restrict__ a, double* __restrict__ b,
                                    int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (double)a[i];
}

__global__ void accumulate_tc_kernel(double* __restrict__ x, const float* __restrict__ dx,
                                     float* __restrict__ x32, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    x[i] += (double)dx[i];
    x32[i] = (float)x[i];
  }
}

// ---------------------------------------------------------------------------
// Preconditioned conjugate gradients for up to kSmallM right-hand sides: the
// FP32 factor L L^T preconditions (K + lambda I) d = r, with x, r, p, q in FP64
// and the products (K + lambda I) v accumulated in double-float. Each column
// stops (its step sizes become 0) once max |r| <= kPcgTol max |b|; when every
// column has stopped the remaining launches return at once.
// ---------------------------------------------------------------------------
constexpr double kPcgTol = 1e-10;   // residual reduction from the starting point
constexpr double kPcgFloor = 1e-15; // or residual below this times max |b|
constexpr int kPcgStall = 2;        // or no halving of the best residual for this many steps
constexpr int kDotBlocks = 304;     // two per SM

struct PcgState {
  double rho[2][kSmallM];   // r.z of the current / next iteration
  double bnorm[kSmallM];    // max |b_j|
  double r0norm[kSmallM];   // max |r_j| of the starting point
  double rbest[kSmallM];    // smallest max |r_j| so far
  int stall[kSmallM];       // iterations since rbest last halved
  double rmax[kSmallM];     // max |r_j| of the last residual
  int active[kSmallM];
  int all_done;
  int ticket;               // blocks of the running kernel that have finished
};

__device__ __forceinline__ void df_add(float& sh, float& sl, float bh, float bl) {
  const float s = sh + bh;
  const float bv = s - sh;
  const float e = (sh - (s - bv)) + (bh - bv);
  sl += e + bl;
  sh = s;
}

// Columns [0, mc) of X (FP64 [n, ldx]) as double-float pairs xs[j, c] = (hi, lo) (pitch
// mc), split once per product so that the row kernel below runs on the FP32 pipes only; x32
// (nullable, pitch mc): their float32 rounding.
__global__ void split_df_kernel(const double* __restrict__ X, int64_t ldx, int64_t n, int64_t mc,
                                float2* __restrict__ xs, float* __restrict__ x32) {
  after_previous();
  const int64_t total = n * mc;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = i / mc, c = i - j * mc;
    const double v = X[j * ldx + c];
    const float h = (float)v;
    xs[i] = make_float2(h, (float)(v - (double)h));
    if (x32) x32[i] = h;
  }
}

// Skinny products with up to MR <= 16 right-hand sides, split along the columns so that
// the grid holds enough tiles to keep every SM busy: tile (rb, kb) covers rows
// [128 rb, 128 rb + 128) and columns [ks kb, ks kb + ks) of M [rows, ncols] (row pitch
// ld, ks a multiple of 32 from split_ks); one thread per row. Each 32-column step of M
// is staged in shared memory from coalesced 16-byte loads (row pitch 33: thread t reads
// its row without bank conflicts), the next step's loads already in flight in registers
// while the current one is multiplied; the matching 32 rows of x are padded to MRP = MR
// rounded up to 4 and read as broadcast 16-byte words. The tile's sums go to
// part[kb][i][c] (FP32) or part2 (double-float pairs); a reduction kernel adds a row's
// tiles in order, so the result does not depend on scheduling. tri 1 (lower: M[i, j] = 0
// for j > i) and 2 (upper: 0 for j < i) skip the tiles outside the triangle. DF: x given
// as its double-float split xs, every product accumulated in double-float (df_fma2: two
// right-hand sides per packed f32x2 instruction); else x FP32 (X) and plain FMA.
template <int MR, bool DF>
__global__ void __launch_bounds__(kGT)
    gemv_part_kernel(const float* __restrict__ M, int64_t ld, int64_t rows, int64_t ncols,
                     int64_t ks, int tri, const float* __restrict__ X,
                     const float2* __restrict__ xs, int64_t m, float* __restrict__ part,
                     float2* __restrict__ part2, const int* skip) {
  after_previous();
  if (skip && *skip) return;
  constexpr int MRP = (MR + 3) & ~3;
  constexpr int NP = (MR + 1) / 2;           // packed column pairs (DF)
  constexpr int NL = kGT * kGK / 4 / kGT;    // 16-byte loads of M per thread and step
  const int64_t r0 = (int64_t)blockIdx.y * kGT, j0 = (int64_t)blockIdx.x * ks;
  if ((tri == 1 && j0 > r0 + kGT - 1) || (tri == 2 && j0 + ks <= r0)) return;
  __shared__ float ms[kGT][kGK + 1];
  __shared__ __align__(16) float xh[kGK][MRP];
  __shared__ __align__(16) float xl[DF ? kGK : 1][DF ? MRP : 4];
  const int t = threadIdx.x;
  // 16-byte loads of M need a pitch of a multiple of 4 floats and an aligned base
  const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(M) & 15) == 0;
  float acc[MR];
  P2 sh2[NP], sl2[NP];
#pragma unroll
  for (int c = 0; c < MR; ++c) acc[c] = 0.f;
#pragma unroll
  for (int q = 0; q < NP; ++q) sh2[q] = sl2[q] = p2s(0.f);
  float4 pre[NL];
  // M[r0 .. r0 + 128)[jb .. jb + 32) into pre: a warp covers 4 rows of 128 bytes
  auto load_step = [&](int64_t jb) {
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int e = t + u * kGT;
      const int64_t row = r0 + (e >> 3), col = jb + (e & 7) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < rows && col < ncols) {
        const float* src = M + row * ld + col;
        if (vec) {
          v = *reinterpret_cast<const float4*>(src);
          // columns beyond ncols (inside the row pitch) are not part of M
          if (col + 1 >= ncols) v.y = 0.f;
          if (col + 2 >= ncols) v.z = 0.f;
          if (col + 3 >= ncols) v.w = 0.f;
        } else {
          v.x = src[0];
          if (col + 1 < ncols) v.y = src[1];
          if (col + 2 < ncols) v.z = src[2];
          if (col + 3 < ncols) v.w = src[3];
        }
      }
      pre[u] = v;
    }
  };
  const int64_t jend = mini(j0 + ks, ncols);
  if (j0 < jend) load_step(j0);
  for (int64_t jb = j0; jb < jend; jb += kGK) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int e = t + u * kGT;
      const int r = e >> 3, j = (e & 7) * 4;
      ms[r][j] = pre[u].x;
      ms[r][j + 1] = pre[u].y;
      ms[r][j + 2] = pre[u].z;
      ms[r][j + 3] = pre[u].w;
    }
    for (int e = t; e < kGK * MRP; e += kGT) {
      const int j = e / MRP, c = e - j * MRP;
      const bool in = jb + j < ncols && c < m;
      if (DF) {
        const float2 v = in ? xs[(jb + j) * m + c] : make_float2(0.f, 0.f);
        xh[j][c] = v.x;
        xl[j][c] = v.y;
      } else {
        xh[j][c] = in ? X[(jb + j) * m + c] : 0.f;
      }
    }
    __syncthreads();
    if (jb + kGK < jend) load_step(jb + kGK);  // in flight during the products below
#pragma unroll 4
    for (int j = 0; j < kGK; ++j) {
      const float a = ms[t][j];
      if (DF) {
        const P2 a2 = p2s(a);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const P2 h = p2ld(&xh[j][2 * q]), l = p2ld(&xl[j][2 * q]);
          df_fma2(a2, h, l, sh2[q], sl2[q]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < MRP / 4; ++q) {
          const float4 h = *reinterpret_cast<const float4*>(&xh[j][4 * q]);
          const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (4 * q + u < MR) acc[4 * q + u] = fmaf(a, hv[u], acc[4 * q + u]);
        }
      }
    }
  }
  const int64_t row = r0 + t;
  if (row >= rows) return;
  const int64_t o = ((int64_t)blockIdx.x * rows + row) * m;
  if (DF) {
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      float h0, h1, l0, l1;
      p2u(sh2[q], h0, h1);
      p2u(sl2[q], l0, l1);
      if (2 * q < m) part2[o + 2 * q] = make_float2(h0, l0);
      if (2 * q + 1 < m) part2[o + 2 * q + 1] = make_float2(h1, l1);
    }
  } else {
#pragma unroll
    for (int c = 0; c < MR; ++c) {
      if (c >= m) break;
      part[o + c] = acc[c];
    }
  }
}

// Column-block width of a split-K product: about `tiles` tiles (1216 tiles of 4 warps:
// 8 resident warps per SM scheduler on 152 SMs; a triangle asks for twice as many, half
// of them lying outside it), a multiple of the 32-column step.
int64_t split_ks(int64_t rows, int64_t ncols, int64_t tiles) {
  const int64_t nrb = ceil_div(rows, kGT);
  const int64_t ks = ceil_div(ceil_div(ncols * nrb, tiles), kGK) * kGK;
  return ks < kGK ? kGK : ks;
}
constexpr int64_t kFullTiles = 1216, kTriTiles = 2432;

// The tiles of a row that gemv_part_kernel computed: [kb_lo, kb_hi).
__device__ __forceinline__ void tile_range(int64_t row, int tri, int ks, int64_t nkb,
                                           int64_t& lo, int64_t& hi) {
  lo = tri == 2 ? row / ks : 0;
  hi = tri == 1 ? row / ks + 1 : nkb;
}

// A block of 256 threads on [rows, m] arrays, m <= kSmallM: cw (the power of two from m on)
// neighbouring threads take a row, so that a thread keeps its column.
struct RowCol {
  int64_t row, step;
  int c;
};
__device__ __forceinline__ RowCol row_col(int64_t m) {
  const int cw = m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : m <= 8 ? 8 : 16, per = 256 / cw;
  return RowCol{(int64_t)blockIdx.x * per + threadIdx.x / cw, (int64_t)gridDim.x * per,
                (int)threadIdx.x % cw};
}
// The block's sums of v by column -> part[block][kSmallM].
__device__ __forceinline__ void column_sums(double v, int64_t m, double* part) {
  __shared__ double red[8][kSmallM];
  const int cw = m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : m <= 8 ? 8 : 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o >= cw; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane < cw) red[warp][lane] = v;
  __syncthreads();
  if (threadIdx.x < m) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w][threadIdx.x];
    part[blockIdx.x * kSmallM + threadIdx.x] = t;
  }
}

// Y[i, c] = sum of the row's tiles, in tile order (FP32 products). Yd, xs (nullable): Y in FP64
// and as a double-float split. r (nullable): the blocks' sums of r_c Y_c into dots. start:
// clears the state for a new iteration.
__global__ void __launch_bounds__(256)
    gemv_reduce_kernel(const float* __restrict__ part, int64_t rows, int64_t m, int tri, int ks,
                       int64_t nkb, float* __restrict__ Y, double* __restrict__ Yd,
                       float2* __restrict__ xs, const double* __restrict__ r,
                       double* __restrict__ dots, PcgState* start, const int* skip) {
  after_previous();
  if (skip && *skip) return;
  if (start && blockIdx.x == 0 && threadIdx.x == 0) start->all_done = start->ticket = 0;
  const RowCol at = row_col(m);
  double d = 0.0;
  for (int64_t row = at.row; row < rows && at.c < m; row += at.step) {
    const int64_t idx = row * m + at.c;
    int64_t lo, hi;
    tile_range(row, tri, ks, nkb, lo, hi);
    float v = 0.f;
#pragma unroll 8
    for (int64_t kb = lo; kb < hi; ++kb) v += part[kb * rows * m + idx];
    Y[idx] = v;
    if (Yd) Yd[idx] = (double)v;
    if (xs) xs[idx] = make_float2(v, 0.f);
    if (r) d = fma(r[idx], (double)v, d);
  }
  if (r) column_sums(d, m, dots);
}

// Double-float products, finished: v = sum of the row's tiles (+ lambda X[i, c] when
// lambda is given: the square (K + lambda I) x), then out = v (mode 0), b - v (mode 1)
// or b + v (mode 2), b = B64 when given, else B (nullable: 0), as FP64 (out) and / or
// FP32 (out32). B, B64, X, out and out32 have row pitch ldo (the tiles' pitch is m). dots
// (nullable): the blocks' sums of X_c v_c.
__global__ void __launch_bounds__(256) df_reduce_kernel(const float2* __restrict__ part2, int64_t rows, int64_t m,
                                 int64_t nkb, const double* lambda, const float* __restrict__ B,
                                 const double* __restrict__ B64, const double* __restrict__ X,
                                 int64_t ldo, int mode,
                                 double* __restrict__ out, float* __restrict__ out32,
                                 double* __restrict__ dots, const int* skip) {
  after_previous();
  if (skip && *skip) return;
  const RowCol at = row_col(m);
  double d = 0.0;
  for (int64_t row = at.row; row < rows && at.c < m; row += at.step) {
    const int64_t idx = row * m + at.c, o = row * ldo + at.c;
    float hi = 0.f, lo = 0.f;
#pragma unroll 4
    for (int64_t kb = 0; kb < nkb; ++kb) {
      const float2 p = part2[kb * rows * m + idx];
      df_add(hi, lo, p.x, p.y);
    }
    double v = (double)hi + (double)lo;
    if (lambda) v += lambda[0] * X[o];
    if (dots) d = fma(X[o], v, d);
    const double b = B64 ? B64[o] : B ? (double)B[o] : 0.0;
    const double r = mode == 1 ? b - v : mode == 2 ? b + v : v;
    if (out) out[o] = r;
    if (out32) out32[o] = (float)r;
  }
  if (dots) column_sums(d, m, dots);
}

template <int MR>
void launch_df_part(cudaStream_t s, dim3 grid, const float* A, int64_t lda, int64_t rows,
                    int64_t ncols, int64_t ks, const float2* xs, int64_t m, float2* part2,
                    const int* skip) {
  launch_next(s, gemv_part_kernel<MR, true>, grid, kGT, A, lda, rows, ncols, ks, 0, nullptr, xs,
              m, nullptr, part2, skip);
}

size_t tri_part_bytes(int64_t n, int64_t m) {
  return (size_t)ceil_div(n, split_ks(n, n, kTriTiles)) * n * m * sizeof(float);
}

size_t df_part_bytes(int64_t rows, int64_t ncols, int64_t m) {
  return (size_t)ceil_div(ncols, split_ks(rows, ncols, kFullTiles)) * rows * m * sizeof(float2);
}

// out = mode(B, (A + [lambda I]) x) for x [ncols, m <= kSmallM] given as its split xs:
// gemv_part_kernel in double-float, then df_reduce_kernel. part2: df_part_bytes.
void launch_matvec(cudaStream_t s, const float* A, int64_t lda, int64_t rows, int64_t ncols,
                   const double* lambda, const float* B, const double* B64, const double* X,
                   const float2* xs,
                   int64_t m, int64_t ldo, int mode, double* out, float* out32, float2* part2,
                   double* dots, const PcgState* st) {
  const int* skip = st ? &st->all_done : nullptr;
  const int64_t ks = split_ks(rows, ncols, kFullTiles), nkb = ceil_div(ncols, ks);
  const dim3 grid((unsigned)nkb, (unsigned)ceil_div(rows, kGT));
  switch (m) {
#define NTG_MV(k) \
  case k: launch_df_part<k>(s, grid, A, lda, rows, ncols, ks, xs, m, part2, skip); break;
    NTG_MV(1) NTG_MV(2) NTG_MV(3) NTG_MV(4) NTG_MV(5) NTG_MV(6) NTG_MV(7) NTG_MV(8)
    NTG_MV(9) NTG_MV(10) NTG_MV(11) NTG_MV(12) NTG_MV(13) NTG_MV(14) NTG_MV(15)
#undef NTG_MV
    default: launch_df_part<kSmallM>(s, grid, A, lda, rows, ncols, ks, xs, m, part2, skip);
  }
  launch_next(s, df_reduce_kernel, dim3(kDotBlocks), 256, part2, rows, m, nkb, lambda, B, B64, X,
              ldo, mode, out, out32, dots, skip);
}

// Sum of the blocks' parts of every column, by the 256 threads of a block -> out[kSmallM].
__device__ __forceinline__ void sum_parts(const double* __restrict__ part, double* out) {
  __shared__ double red[16][kSmallM];
  const int c = threadIdx.x & 15, g = threadIdx.x >> 4;
  double t = 0.0;
#pragma unroll
  for (int b = g; b < kDotBlocks; b += 16) t += part[b * kSmallM + c];
  red[g][c] = t;
  __syncthreads();
  if (threadIdx.x < kSmallM) {
    t = 0.0;
    for (int w = 0; w < 16; ++w) t += red[w][threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// Whether this block is the last of the grid to get here; its view of the others' writes is
// then complete.
__device__ __forceinline__ bool last_block(PcgState* st) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// The maxima of non-negative values are taken on their 64-bit patterns, where a NaN is the
// largest. max_parts: over all blocks' parts of every column, by the 256 threads of a block.
__device__ __forceinline__ double pattern_max(double a, double b) {
  return __double_as_longlong(a) > __double_as_longlong(b) ? a : b;
}

__device__ __forceinline__ void max_parts(const double* part, double* out) {
  __shared__ double red[16][kSmallM];
  const int c = threadIdx.x & 15, g = threadIdx.x >> 4;
  double t = 0.0;
  for (int b = g; b < (int)gridDim.x; b += 16)
    t = pattern_max(t, *reinterpret_cast<const volatile double*>(part + b * kSmallM + c));
  red[g][c] = t;
  __syncthreads();
  if (threadIdx.x < kSmallM) {
    for (int w = 0; w < 16; ++w) t = pattern_max(t, red[w][threadIdx.x]);
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

__device__ __forceinline__ void block_max(double* slot, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(slot),
            (unsigned long long)__double_as_longlong(fabs(v)));
}

// With the sums, splits and checks of an iteration in the kernels next to them and every launch
// set up under the one before (launch_next), 5000 points and ten right-hand sides take 245 us
// an iteration (290 in twelve plain launches), an iteration after convergence, eight kernels
// that return at once, 14 us (48).

// Set-up: p = z and its split; bnorm, r0norm, rho[0] = r.z (from part), every column active.
// bpart, rpart: the blocks' maxima.
__global__ void __launch_bounds__(256)
    pcg_init_kernel(const float* __restrict__ B, const float* __restrict__ z,
                    double* __restrict__ p, float2* __restrict__ xs, const double* __restrict__ r,
                    int64_t n, int64_t m, const double* __restrict__ part, double* bpart,
                    double* rpart, PcgState* st) {
  after_previous();
  __shared__ double bmax[kSmallM], rmax[kSmallM], rho[kSmallM];
  if (threadIdx.x < kSmallM) bmax[threadIdx.x] = rmax[threadIdx.x] = 0.0;
  __syncthreads();
  const RowCol at = row_col(m);
  double bm = 0.0, rm = 0.0;
  for (int64_t row = at.row; row < n && at.c < m; row += at.step) {
    const int64_t i = row * m + at.c;
    p[i] = (double)z[i];
    xs[i] = make_float2(z[i], 0.f);
    bm = pattern_max(bm, fabs((double)B[i]));
    rm = pattern_max(rm, fabs(r[i]));
  }
  if (at.c < m) {
    block_max(&bmax[at.c], bm);
    block_max(&rmax[at.c], rm);
  }
  __syncthreads();
  if (threadIdx.x < kSmallM) {
    bpart[blockIdx.x * kSmallM + threadIdx.x] = bmax[threadIdx.x];
    rpart[blockIdx.x * kSmallM + threadIdx.x] = rmax[threadIdx.x];
  }
  if (!last_block(st)) return;
  max_parts(bpart, bmax);
  max_parts(rpart, rmax);
  sum_parts(part, rho);
  if (threadIdx.x < m) {
    const int c = threadIdx.x;
    st->bnorm[c] = bmax[c];
    st->r0norm[c] = rmax[c];
    st->rbest[c] = rmax[c];
    st->stall[c] = 0;
    st->rho[0][c] = rho[c];
    st->rmax[c] = rmax[c];
    st->active[c] = rmax[c] > kPcgFloor * bmax[c];
  }
  if (threadIdx.x == 0) st->ticket = 0;
}

// x += alpha p, r -= alpha q (alpha_c = rho_c / p.q), r32 = (float) r; then, in the last
// block, the convergence of each column by max |r_c|: one at or below kPcgTol max |b_c|
// stops; all_done once none is left.
__global__ void __launch_bounds__(256)
    pcg_step_kernel(double* __restrict__ x, double* __restrict__ r, float* __restrict__ r32,
                    const double* __restrict__ p, const double* __restrict__ q, int64_t n,
                    int64_t m, const double* __restrict__ pq_part, double* rpart, PcgState* st,
                    int cur) {
  after_previous();
  if (st->all_done) return;
  __shared__ double pq[kSmallM], rmax[kSmallM];
  __shared__ int any;
  if (threadIdx.x < kSmallM) rmax[threadIdx.x] = 0.0;
  if (threadIdx.x == 0) any = 0;
  sum_parts(pq_part, pq);
  const RowCol at = row_col(m);
  double rm = 0.0;
  if (at.c < m) {
    const int c = at.c;
    const double a = (st->active[c] && pq[c] > 0.0) ? st->rho[cur][c] / pq[c] : 0.0;
    for (int64_t row = at.row; row < n; row += at.step) {
      const int64_t i = row * m + c;
      x[i] = fma(a, p[i], x[i]);
      const double rv = fma(-a, q[i], r[i]);
      r[i] = rv;
      r32[i] = (float)rv;
      rm = pattern_max(rm, fabs(rv));
    }
    block_max(&rmax[c], rm);
  }
  __syncthreads();
  if (threadIdx.x < kSmallM) rpart[blockIdx.x * kSmallM + threadIdx.x] = rmax[threadIdx.x];
  if (!last_block(st)) return;
  max_parts(rpart, rmax);
  if (threadIdx.x < m) {
    const int c = threadIdx.x;
    const double mx = rmax[c];
    st->rmax[c] = mx;
    // the double-float products put a floor under the residual: a column whose best
    // residual has not halved in kPcgStall iterations has reached it and stops
    if (mx < 0.5 * st->rbest[c]) {
      st->rbest[c] = mx;
      st->stall[c] = 0;
    } else {
      ++st->stall[c];
    }
    if (st->active[c] && (mx <= kPcgTol * st->r0norm[c] || mx <= kPcgFloor * st->bnorm[c] ||
                          st->stall[c] >= kPcgStall))
      st->active[c] = 0;
    if (st->active[c]) atomicOr(&any, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    st->ticket = 0;
    if (!any) st->all_done = 1;
  }
}

// beta_c = (r.z)_new / rho_c; p = z + beta p and its split; rho[nxt] = (r.z)_new.
__global__ void __launch_bounds__(256)
    pcg_dir_kernel(double* __restrict__ p, float2* __restrict__ xs, const float* __restrict__ z,
                   int64_t n, int64_t m, const double* __restrict__ rz_part, PcgState* st,
                   int cur) {
  after_previous();
  if (st->all_done) return;
  __shared__ double rz[kSmallM];
  sum_parts(rz_part, rz);
  const int nxt = cur ^ 1;
  const RowCol at = row_col(m);
  if (at.c >= m) return;
  const double beta = st->rho[cur][at.c] != 0.0 ? rz[at.c] / st->rho[cur][at.c] : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == at.c) st->rho[nxt][at.c] = rz[at.c];
  if (!st->active[at.c]) return;
  for (int64_t row = at.row; row < n; row += at.step) {
    const int64_t i = row * m + at.c;
    const double v = fma(beta, p[i], (double)z[i]);
    p[i] = v;
    const float h = (float)v;
    xs[i] = make_float2(h, (float)(v - (double)h));
  }
}

__global__ void logdet_ld_kernel(const float* __restrict__ L, int64_t n, int64_t ldl,
                                 double* __restrict__ out) {
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += log((double)L[i * ldl + i]);
  __shared__ double part[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    out[0] = 2.0 * t;
  }
}


int set_smem(const void* fn, size_t bytes) {
  const cudaError_t e =
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return fail(NTG_ERR_CUDA, std::string("chol: ") + cudaGetErrorString(e));
  return NTG_OK;
}

int attrs_once() {
  static std::once_flag once;
  static int rc = NTG_OK;
  std::call_once(once, [] {
    rc = set_smem((const void*)diag_block_kernel, kDiagSmem);
  });
  return rc;
}

// Per-device streams and events of the factorisation: the critical chain (diagonal block,
// next_tile_kernel) and, beside it, the rest of the panel and of the next column block on
// high-priority streams, the bulk of each trailing update on a third stream one panel behind
// them, and the inverse factor L^-T, block by block as the panels become final, on a fourth.
struct SideStream {
  cudaStream_t hi = nullptr, near = nullptr, trail = nullptr, side = nullptr;
  cudaEvent_t fork = nullptr, diag = nullptr, next = nullptr, panel = nullptr, column = nullptr,
              trail_done = nullptr;
  cudaEvent_t join[4] = {nullptr, nullptr, nullptr, nullptr};
  // held while one factorisation enqueues its work: the events are re-recorded per panel,
  // and two host threads interleaving their records and waits would order each other's
  // launches (a wait, once enqueued, is not affected by a later record)
  std::mutex enqueue;
};

int side_stream(SideStream** out) {
  static std::mutex mu;
  static SideStream per_dev[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return fail(NTG_ERR_CUDA, "chol: no current device");
  std::lock_guard<std::mutex> lock(mu);
  SideStream& ss = per_dev[dev];
  if (!ss.hi) {
    int least = 0, greatest = 0;
    bool ok = cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess;
    ok = ok && cudaStreamCreateWithPriority(&ss.hi, cudaStreamNonBlocking, greatest) == cudaSuccess;
    ok = ok && cudaStreamCreateWithPriority(&ss.near, cudaStreamNonBlocking, greatest) == cudaSuccess;
    ok = ok && cudaStreamCreateWithPriority(&ss.trail, cudaStreamNonBlocking, least) == cudaSuccess;
    ok = ok && cudaStreamCreateWithPriority(&ss.side, cudaStreamNonBlocking, least) == cudaSuccess;
    cudaEvent_t* evs[10] = {&ss.fork,       &ss.diag,    &ss.next,    &ss.panel,   &ss.column,
                            &ss.trail_done, &ss.join[0], &ss.join[1], &ss.join[2], &ss.join[3]};
    for (cudaEvent_t* e : evs)
      ok = ok && cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
      ss.hi = nullptr;
      return fail(NTG_ERR_CUDA, "chol: stream creation failed");
    }
  }
  *out = &ss;
  return NTG_OK;
}

// Factor workspace layout: linv [nblk * 128 * 128] f32 (inverses of the diagonal
// blocks), uinv = L^-T [n * ldl] f32 (upper), linvf = L^-1 [n * ldl] f32 (lower).
struct FactorWs {
  float* linv;
  float* uinv;
  float* linvf;
};

size_t factor_ws_bytes(int64_t n, int64_t ldl) {
  const int64_t nblk = (n + PB - 1) / PB;
  return (size_t)(nblk * PB * PB + 2 * n * ldl) * sizeof(float) + 256;
}

FactorWs factor_ws(void* ws, int64_t n, int64_t ldl) {
  const int64_t nblk = (n + PB - 1) / PB;
  char* p = static_cast<char*>(ws);
  p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 255) & ~(uintptr_t)255);
  FactorWs f;
  f.linv = reinterpret_cast<float*>(p);
  f.uinv = f.linv + nblk * PB * PB;
  f.linvf = f.uinv + n * ldl;
  return f;
}

// Solve workspace: rnorm (256 B), x64 [n m] f64, r32 [n m] f32, t32 [n m] f32, then
// for m <= kSmallM the PCG vectors r64, p64, q64 [n m] f64, three dot-product partial
// arrays [kDotBlocks * kSmallM] f64, the PcgState and the double-float split of the
// current vector [n m] float2, and the split-K tiles of the triangular and double-float
// products; for more, z [m * ldl] f32, y [m * ldl] f32 (the transposed right-hand sides
// and their half-solved form) and the double-float split of x [n m] float2, or the digits
// of the exact residual.
size_t solve_ws_bytes(int64_t n, int64_t m, int64_t ldl) {
  size_t b = 256 + (size_t)n * m * (sizeof(double) + 2 * sizeof(float)) + 256;
  if (m > kSmallM)
    b += 2 * (size_t)m * ldl * sizeof(float) + 512 +
         (exact_residual_pays(n, m) ? exact_residual_bytes(n, m) : (size_t)n * m * sizeof(float2));
  else b += (size_t)3 * n * m * sizeof(double) + 3 * kDotBlocks * kSmallM * sizeof(double) +
            sizeof(PcgState) + 256 + (size_t)n * m * sizeof(float2) + 256 +
            tri_part_bytes(n, m) + 256 + df_part_bytes(n, n, m) + 256;
  return (b + 255) & ~(size_t)255;
}

// X = (L L^T)^-1 X for up to kSmallM right-hand sides: t = L^-1 X, X = L^-T t, each a
// split-K triangular product (gemv_part_kernel) and its reduction; tpart holds
// tri_part_bytes(n, m). Xd, xs, r, dots, start: of the last reduction (gemv_reduce_kernel).
template <int MR>
void launch_tri_part(cudaStream_t s, dim3 grid, const float* M, int64_t ld, int64_t n,
                     int64_t ks, int tri, const float* X, int64_t m, float* part,
                     const int* skip) {
  launch_next(s, gemv_part_kernel<MR, false>, grid, kGT, M, ld, n, n, ks, tri, X, nullptr, m,
              part, nullptr, skip);
}

int inv_apply_small(cudaStream_t s, const FactorWs& f, int64_t ldl, int64_t n, float* X, int64_t m,
                    float* t, float* tpart, const int* skip, double* Xd = nullptr,
                    float2* xs = nullptr, const double* r = nullptr, double* dots = nullptr,
                    PcgState* start = nullptr) {
  const int64_t ks = split_ks(n, n, kTriTiles), nkb = ceil_div(n, ks);
  const dim3 grid((unsigned)nkb, (unsigned)ceil_div(n, kGT));
  auto tri = [&](const float* M, int tri, const float* in, float* out) {
    if (m == 1) launch_tri_part<1>(s, grid, M, ldl, n, ks, tri, in, m, tpart, skip);
    else if (m <= 4) launch_tri_part<4>(s, grid, M, ldl, n, ks, tri, in, m, tpart, skip);
    else if (m <= 10) launch_tri_part<10>(s, grid, M, ldl, n, ks, tri, in, m, tpart, skip);
    else launch_tri_part<kSmallM>(s, grid, M, ldl, n, ks, tri, in, m, tpart, skip);
    const bool last = tri == 2;
    launch_next(s, gemv_reduce_kernel, dim3(kDotBlocks), 256, tpart, n, m, tri, (int)ks, nkb, out,
                last ? Xd : nullptr, last ? xs : nullptr, last ? r : nullptr, dots,
                last ? start : nullptr, skip);
  };
  tri(f.linvf, 1, X, t);  // L^-1: lower
  tri(f.uinv, 2, t, X);   // L^-T: upper
  return check_launch("ntg_chol_solve_tc apply");
}

// X = (L L^T)^-1 X for many right-hand sides on the tensor cores, through the transposed
// right-hand sides z = X^T [m, ldl]: y = z L^-T (= (L^-1 X)^T), z = y L^-1 (= X'^T). Each
// tile's sum runs over the triangle only (4096 right-hand sides, n 4096: 907 -> 470 us a
// product, 393 since the split has eight warps).
int inv_apply_many(cudaStream_t s, const FactorWs& f, int64_t ldl, int64_t n, float* X, int64_t m,
                   float* z, float* y) {
  {
    dim3 g((unsigned)ceil_div(m, 32), (unsigned)ceil_div(n, 32));
    transpose_kernel<<<g, 256, 0, s>>>(X, m, z, ldl, n, m, false);
    note_launch();
  }
  // y[c, j] = sum_i z[c, i] L^-1[j, i]: NT with B = L^-1 (row-major)
  int rc = gemm_tf32x3(s, z, ldl, f.linvf, ldl, y, ldl, m, n, n, 1.f, 0.f, 0, 1);
  if (rc) return rc;
  // z[c, i] = sum_j y[c, j] L^-T[i, j]: NT with B = L^-T (row-major)
  rc = gemm_tf32x3(s, y, ldl, f.uinv, ldl, z, ldl, m, n, n, 1.f, 0.f, 0, 2);
  if (rc) return rc;
  {
    dim3 g((unsigned)ceil_div(n, 32), (unsigned)ceil_div(m, 32));
    transpose_kernel<<<g, 256, 0, s>>>(z, ldl, X, m, m, n, false);
    note_launch();
  }
  return check_launch("ntg_chol_solve_tc apply");
}

}  // namespace

}  // namespace ntg

using namespace ntg;

extern "C" size_t ntg_chol_factor_tc_workspace_bytes(int64_t n, int64_t ldl) {
  if (n <= 0 || ldl < n || n > 46340 || ldl > 46340 + 128) return SIZE_MAX;
  return factor_ws_bytes(n, ldl);
}

extern "C" int ntg_chol_factor_tc(void* stream, const float* A, int64_t n, double diag_reg,
                                  int32_t absolute, float* L, int64_t ldl, double* lambda,
                                  int* info, void* workspace, size_t workspace_bytes) {
  NTG_REQUIRE(A && L && lambda && info && workspace, "ntg_chol_factor_tc: null pointer");
  NTG_REQUIRE(n > 0 && n <= 46340, "ntg_chol_factor_tc: n must be in [1, 46340]");
  NTG_REQUIRE(ldl >= n && ldl % 4 == 0 && ldl <= 46340 + 128,
              "ntg_chol_factor_tc: ldl must be >= n and a multiple of 4");
  NTG_REQUIRE((reinterpret_cast<uintptr_t>(L) & 15) == 0, "ntg_chol_factor_tc: L must be 16-byte aligned");
  NTG_REQUIRE(workspace_bytes >= factor_ws_bytes(n, ldl),
              "ntg_chol_factor_tc: workspace smaller than ntg_chol_factor_tc_workspace_bytes");
  int rc = attrs_once();
  if (rc) return rc;
  cudaStream_t s = as_stream(stream);
  const FactorWs f = factor_ws(workspace, n, ldl);
  if (cudaMemsetAsync(info, 0, sizeof(int), s) != cudaSuccess)
    return check_launch("ntg_chol_factor_tc memset");
  trace_tc_kernel<<<1, 1024, 0, s>>>(A, n, lambda + 1);
  init_factor_ld_kernel<<<dim3((unsigned)ceil_div(ldl, 1024), (unsigned)n), 256, 0, s>>>(
      A, n, ldl, diag_reg, absolute, lambda + 1, L, f.uinv, lambda);
  note_launch(2);
  SideStream* ss = nullptr;
  rc = side_stream(&ss);
  if (rc) return rc;
  std::lock_guard<std::mutex> enqueue_lock(ss->enqueue);
  // L^-T by the forward block solve of L Y = I on the transposed side, Z = Y^T: per
  // block b, Z[:, b] <- Z[:, b] Linv_b^T, then Z[:, >b] -= Z[:, b] L[>b, b]^T, where only
  // the rows [0, r0 + nb) of Z[:, b] are non-zero (Z is upper triangular). Step b reads
  // panel b and Linv_b only, which no later panel changes.
  auto record_wait = [](cudaEvent_t e, cudaStream_t from, cudaStream_t to) {
    return cudaEventRecord(e, from) == cudaSuccess && cudaStreamWaitEvent(to, e, 0) == cudaSuccess;
  };
  if (!record_wait(ss->fork, s, ss->hi) || cudaStreamWaitEvent(ss->trail, ss->fork, 0) ||
      cudaStreamWaitEvent(ss->side, ss->fork, 0) || cudaStreamWaitEvent(ss->near, ss->fork, 0))
    return check_launch("ntg_chol_factor_tc fork");
  // every return after the fork joins the four streams back into s
  auto join = [&]() -> int {
    const cudaStream_t from[4] = {ss->hi, ss->near, ss->trail, ss->side};
    for (int i = 0; i < 4; ++i)
      if (!record_wait(ss->join[i], from[i], s)) return check_launch("ntg_chol_factor_tc join");
    return NTG_OK;
  };
  auto wait = [](cudaStream_t to, cudaEvent_t e) {
    return cudaStreamWaitEvent(to, e, 0) == cudaSuccess;
  };
  // Step b. hi: diagonal block b, then the tile of L21 and the update (next_tile_kernel) that
  // block b + 1 waits for. near: the rows of the panel and of column block b + 1 below these.
  // trail: the columns beyond (rows and columns >= k + 2 PB). Column block b + 1 and block
  // (b + 1, b + 1) come after the trailing update of panel b - 1, which also wrote them.
  const int64_t nblk = (n + PB - 1) / PB;
  for (int64_t b = 0; b < nblk; ++b) {
    const int64_t k = b * PB;
    float* const linv = f.linv + b * PB * PB;
    const int64_t rest = n - k - PB, nb1 = mini(PB, rest), far = rest - nb1;
    float* const l21 = L + (k + PB) * ldl + k;  // rows of the next block
    float* const l31 = l21 + PB * ldl;          // rows beyond
    bool ok = true;
    launch_next_smem(ss->hi, diag_block_kernel, dim3(1), 512, kDiagSmem, L, ldl, n, k, info, linv);
    if (rest > 0) {
      ok = record_wait(ss->diag, ss->hi, ss->near);
      if (b > 0) ok = ok && wait(ss->hi, ss->column) && wait(ss->hi, ss->trail_done);
      launch_next(ss->hi, next_tile_kernel<false>, dim3(PB / 16), 256, L, ldl, n, k, linv);
      launch_next(ss->hi, next_tile_kernel<true>, dim3(PB / 16), 256, L, ldl, n, k, linv);
    }
    ok = ok && record_wait(ss->next, ss->hi, ss->side);
    if (!ok) return join(), check_launch("ntg_chol_factor_tc events");
    if (far > 0) {
      // in place (n = 128 columns: each tile row is read before it is written)
      rc = gemm_tf32x3(ss->near, l31, ldl, linv, PB, l31, ldl, far, PB, PB, 1.f, 0.f, 0);
      if (rc) return join(), rc;
      ok = record_wait(ss->panel, ss->near, ss->side) && wait(ss->trail, ss->panel) &&
           wait(ss->near, ss->next) && (b == 0 || wait(ss->near, ss->trail_done));
      if (!ok) return join(), check_launch("ntg_chol_factor_tc events");
      rc = gemm_tf32x3(ss->near, l31, ldl, l21, ldl, L + (k + 2 * PB) * ldl + k + PB, ldl, far,
                       nb1, PB, -1.f, 1.f, 0);
      if (rc) return join(), rc;
      rc = gemm_tf32x3(ss->trail, l31, ldl, l31, ldl, L + (k + 2 * PB) * ldl + k + 2 * PB, ldl, far,
                       far, PB, -1.f, 1.f, 1);
      if (rc) return join(), rc;
      if (cudaEventRecord(ss->column, ss->near) != cudaSuccess ||
          cudaEventRecord(ss->trail_done, ss->trail) != cudaSuccess)
        return join(), check_launch("ntg_chol_factor_tc events");
    }
    const int64_t nb = mini(PB, n - k), rows = k + nb;
    rc = gemm_tf32x3(ss->side, f.uinv + k, ldl, linv, PB, f.uinv + k, ldl, rows, nb, nb, 1.f, 0.f,
                     0);
    if (rc) return join(), rc;
    if (n - rows > 0) {
      rc = gemm_tf32x3(ss->side, f.uinv + k, ldl, L + rows * ldl + k, ldl, f.uinv + rows, ldl, rows,
                       n - rows, nb, -1.f, 1.f, 0);
      if (rc) return join(), rc;
    }
  }
  rc = join();
  if (rc) return rc;
  dim3 g((unsigned)ceil_div(n, 32), (unsigned)ceil_div(n, 32));
  transpose_kernel<<<g, 256, 0, s>>>(f.uinv, ldl, f.linvf, ldl, n, n, true);
  note_launch();
  return check_launch("ntg_chol_factor_tc");
}

extern "C" size_t ntg_chol_solve_tc_workspace_bytes(int64_t n, int64_t m, int64_t ldl) {
  if (n <= 0 || m <= 0 || ldl < n || n > 46340) return SIZE_MAX;
  const uint64_t per = sizeof(double) + sizeof(float) + sizeof(float);
  if ((uint64_t)m > ((uint64_t)INT64_MAX / per) / (uint64_t)ldl) return SIZE_MAX;
  return solve_ws_bytes(n, m, ldl);
}

extern "C" int ntg_chol_solve_tc(void* stream, const float* A, const float* L, int64_t ldl,
                                 const void* factor_workspace, const double* lambda, int64_t n,
                                 const float* B, int64_t m, float* X, int32_t refine_iters,
                                 void* workspace, size_t workspace_bytes,
                                 double* final_residual, double* x64_out, const double* B64) {
  NTG_REQUIRE(A && L && factor_workspace && lambda && B && X && workspace,
              "ntg_chol_solve_tc: null pointer");
  NTG_REQUIRE(n > 0 && n <= 46340 && m > 0, "ntg_chol_solve_tc: bad sizes");
  NTG_REQUIRE(ldl >= n && ldl % 4 == 0, "ntg_chol_solve_tc: bad ldl");
  NTG_REQUIRE(refine_iters >= 0 && refine_iters <= 64, "ntg_chol_solve_tc: 0..64 refinement steps");
  NTG_REQUIRE(m <= (1ll << 31) / 64, "ntg_chol_solve_tc: too many right-hand sides");
  NTG_REQUIRE(workspace_bytes >= ntg_chol_solve_tc_workspace_bytes(n, m, ldl),
              "ntg_chol_solve_tc: workspace smaller than ntg_chol_solve_tc_workspace_bytes");
  (void)L;  // the solves use the inverse factors kept in factor_workspace
  int rc = attrs_once();
  if (rc) return rc;
  cudaStream_t s = as_stream(stream);
  const FactorWs f = factor_ws(const_cast<void*>(factor_workspace), n, ldl);
  char* ws = static_cast<char*>(workspace);
  double* rnorm = reinterpret_cast<double*>(ws);
  double* x64 = reinterpret_cast<double*>(ws + 256);
  float* r32 = reinterpret_cast<float*>(x64 + n * m);
  float* t32 = r32 + n * m;
  char* tail = reinterpret_cast<char*>(
      (reinterpret_cast<uintptr_t>(t32 + n * m) + 255) & ~(uintptr_t)255);
  float* z = reinterpret_cast<float*>(tail);
  float* y = reinterpret_cast<float*>(
      (reinterpret_cast<uintptr_t>(z + m * ldl) + 255) & ~(uintptr_t)255);
  auto align256 = [](const void* p) {
    return reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 255) & ~(uintptr_t)255);
  };
  // m <= kSmallM: the PCG vectors and the products' split-K tiles
  double* r64 = reinterpret_cast<double*>(tail);
  double* p64 = r64 + n * m;
  double* q64 = p64 + n * m;
  double* part = q64 + n * m;
  double* part_rz = part + kDotBlocks * kSmallM;
  double* part_r = part_rz + kDotBlocks * kSmallM;
  PcgState* st = reinterpret_cast<PcgState*>(part_r + kDotBlocks * kSmallM);
  float2* xs = reinterpret_cast<float2*>(align256(st + 1));
  float* tpart = reinterpret_cast<float*>(align256(xs + n * m));
  float2* dpart = reinterpret_cast<float2*>(align256(reinterpret_cast<char*>(tpart) +
                                                     tri_part_bytes(n, m)));
  if (cudaMemcpyAsync(X, B, sizeof(float) * n * m, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return check_launch("ntg_chol_solve_tc copy");
  const bool few = m <= kSmallM, only = refine_iters == 0 && !final_residual;
  rc = few ? inv_apply_small(s, f, ldl, n, X, m, t32, tpart, nullptr, only ? x64_out : x64,
                             only ? nullptr : xs)
           : inv_apply_many(s, f, ldl, n, X, m, z, y);
  if (rc) return rc;
  if (!few) {
    double* const xd = only ? x64_out : x64;
    if (xd) {
      to_double_tc_kernel<<<grid_for(n * m), 256, 0, s>>>(X, xd, n * m);
      note_launch();
    }
  }
  if (only) return check_launch("ntg_chol_solve_tc");
  // the FP64 solution, for products that must keep its precision (ntg_gemm_df)
  auto copy_x64 = [&]() -> int {
    if (x64_out && cudaMemcpyAsync(x64_out, x64, sizeof(double) * n * m,
                                   cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return check_launch("ntg_chol_solve_tc solution copy");
    return NTG_OK;
  };
  if (few) {
    // preconditioned conjugate gradients on (K + lambda I) x = b from x0 = (L L^T)^-1 b;
    // (K + lambda I) v for v = x64 or p64 (subtract: b - ...), through the split of v in xs,
    // which the kernel that wrote v has left there
    auto matvec = [&](const double* v, int subtract, const float* bb, double* out, float* o32,
                      double* dots, const PcgState* stp) {
      launch_matvec(s, A, n, n, n, lambda, bb, bb ? B64 : nullptr, v, xs, m, m, subtract, out, o32,
                    dpart, dots, stp);
    };
    if (refine_iters > 0) {
      matvec(x64, 1, B, r64, r32, nullptr, nullptr);
      rc = inv_apply_small(s, f, ldl, n, r32, m, t32, tpart, nullptr, nullptr, nullptr, r64,
                           part_rz, st);  // z0
      if (rc) return rc;
      launch_next(s, pcg_init_kernel, dim3(kDotBlocks), 256, B, r32, p64, xs, r64, n, m, part_rz,
                  part, part_r, st);
      for (int it = 0; it < refine_iters; ++it) {
        const int cur = it & 1;
        matvec(p64, 0, nullptr, q64, nullptr, part, st);
        launch_next(s, pcg_step_kernel, dim3(kDotBlocks), 256, x64, r64, r32, p64, q64, n, m, part,
                    part_r, st, cur);
        rc = inv_apply_small(s, f, ldl, n, r32, m, t32, tpart, &st->all_done, nullptr, nullptr,
                             r64, part_rz);
        if (rc) return rc;
        launch_next(s, pcg_dir_kernel, dim3(kDotBlocks), 256, p64, xs, r32, n, m, part_rz, st,
                    cur);
      }
      launch_next(s, split_df_kernel, dim3(grid_for(n * m)), 256, x64, m, n, m, xs, X);
    }
    if (final_residual) {
      // the true residual of the returned solution
      matvec(x64, 1, B, r64, nullptr, nullptr, nullptr);
      if (cudaMemsetAsync(rnorm, 0, sizeof(double), s) != cudaSuccess)
        return check_launch("ntg_chol_solve_tc memset");
      max_abs64_kernel<<<grid_for(n * m), 256, 0, s>>>(r64, n * m, rnorm);
      note_launch();
      if (cudaMemcpyAsync(final_residual, rnorm, sizeof(double), cudaMemcpyDeviceToDevice, s) !=
          cudaSuccess)
        return check_launch("ntg_chol_solve_tc residual copy");
    }
    rc = copy_x64();
    if (rc) return rc;
    return check_launch("ntg_chol_solve_tc");
  }
  // many right-hand sides: refine_iters steps of iterative refinement
  float2* xsplit = reinterpret_cast<float2*>(align256(y + m * ldl));
  for (int it = 0; it <= refine_iters; ++it) {
    if (it == refine_iters && !final_residual) break;
    if (cudaMemsetAsync(rnorm, 0, sizeof(double), s) != cudaSuccess)
      return check_launch("ntg_chol_solve_tc memset");
    if (exact_residual_pays(n, m)) {
      rc = exact_residual(s, A, n, lambda, B, B64, x64, m, r32, rnorm, xsplit, it > 0);
      if (rc) return rc;
    } else {
      launch_next(s, split_df_kernel, dim3(grid_for(n * m)), 256, x64, m, n, m, xsplit, nullptr);
      residual_df_kernel<<<dim3((unsigned)ceil_div(m, 64), (unsigned)ceil_div(n, 64)), 256, 0, s>>>(
          A, n, lambda, B, B64, x64, xsplit, m, r32, rnorm);
      note_launch();
    }
    if (it == refine_iters) break;
    rc = inv_apply_many(s, f, ldl, n, r32, m, z, y);
    if (rc) return rc;
    accumulate_tc_kernel<<<grid_for(n * m), 256, 0, s>>>(x64, r32, X, n * m);
    note_launch();
  }
  if (final_residual &&
      cudaMemcpyAsync(final_residual, rnorm, sizeof(double), cudaMemcpyDeviceToDevice, s) !=
          cudaSuccess)
    return check_launch("ntg_chol_solve_tc residual copy");
  rc = copy_x64();
  if (rc) return rc;
  return check_launch("ntg_chol_solve_tc");
}

extern "C" size_t ntg_gemm_df_workspace_bytes(int64_t rows, int64_t n, int64_t m) {
  if (rows <= 0 || n <= 0 || m <= 0) return SIZE_MAX;
  const int64_t mc = mini(m, kSmallM);
  return (size_t)n * mc * sizeof(float2) + 256 + df_part_bytes(rows, n, mc) + 256;
}

extern "C" int ntg_gemm_df(void* stream, const float* A, int64_t lda, int64_t rows, int64_t n,
                           const double* X, int64_t m, const float* Y0, float* Y, double* Y64,
                           void* workspace, size_t workspace_bytes) {
  NTG_REQUIRE(A && X && (Y || Y64) && workspace, "ntg_gemm_df: null pointer");
  NTG_REQUIRE(rows > 0 && n > 0 && m > 0 && lda >= n, "ntg_gemm_df: bad sizes");
  NTG_REQUIRE(workspace_bytes >= ntg_gemm_df_workspace_bytes(rows, n, m),
              "ntg_gemm_df: workspace smaller than ntg_gemm_df_workspace_bytes");
  cudaStream_t s = as_stream(stream);
  float2* xs = reinterpret_cast<float2*>(
      (reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255);
  float2* dpart = reinterpret_cast<float2*>(
      (reinterpret_cast<uintptr_t>(xs + n * mini(m, kSmallM)) + 255) & ~(uintptr_t)255);
  for (int64_t c0 = 0; c0 < m; c0 += kSmallM) {
    const int64_t mc = mini(kSmallM, m - c0);
    launch_next(s, split_df_kernel, dim3(grid_for(n * mc)), 256, X + c0, m, n, mc, xs, nullptr);
    launch_matvec(s, A, lda, rows, n, nullptr, Y0 ? Y0 + c0 : nullptr, nullptr, nullptr, xs, mc,
                  m, 2, Y64 ? Y64 + c0 : nullptr, Y ? Y + c0 : nullptr, dpart, nullptr, nullptr);
  }
  return check_launch("ntg_gemm_df");
}

extern "C" int ntg_chol_logdet_tc(void* stream, const float* L, int64_t n, int64_t ldl,
                                  double* out) {
  NTG_REQUIRE(L && out && n > 0 && ldl >= n, "ntg_chol_logdet_tc: bad arguments");
  logdet_ld_kernel<<<1, 1024, 0, as_stream(stream)>>>(L, n, ldl, out);
  note_launch();
  return check_launch("ntg_chol_logdet_tc");
}
