// Symmetric eigendecomposition for the finite-time predictions of
// predict.gradient_descent_mse and gradient_descent_mse_ensemble
// (neural_tangents/_src/predict.py:185-229, 1180-1221, where the reference calls
// eigh): two-sided block Jacobi in FP32.
//
// The matrix (padded with zeros to a multiple of 64; padded indices never couple
// to the others, so they stay exact unit vectors) is split into 32-wide blocks.
// A sweep pairs every two blocks once, in the round-robin order of a tournament
// (nb - 1 rounds of nb / 2 disjoint pairs). In a round:
//   jacobi_inner_kernel   one CTA per pair runs a sweep of cyclic parallel
//                         Jacobi on the 64 x 64 matrix of its two blocks in shared
//                         memory (over the couplings between the blocks; over all in
//                         the first round) and writes the accumulated rotation U (64 x 64);
//                         what couplings remain stay in A for the next sweeps;
//   jacobi_apply_kernel   A <- U^T A U tile by tile (a 64 x 64 tile of A couples
//                         two pairs and depends only on their rotations) and V <- V U.
// After each sweep off(A) / ||A||_F is read back (one 16-byte copy) and the sweeps
// stop below the tolerance (or when rounding stops them). Eigenvalues are the diagonal of the final A, not sorted.
// FP32 rounding accumulates over the rounds (about 1e-5 relative at n = 1000), so the
// pairs are then refined with double-float products (see the refinement below).
#include <cmath>
#include <string>
#include <vector>

#include "ntg_common.cuh"

namespace ntg {
namespace {

constexpr int JB = 32;        // block width
constexpr int JP = 2 * JB;    // a pair: 64 indices

__host__ __device__ __forceinline__ void rr_pair(int nplayers, int round, int k, int& a, int& b) {
  // circle method: player nplayers - 1 fixed, the others rotate
  const int m = nplayers - 1;
  if (k == 0) {
    a = m;
    b = round % m;
  } else {
    a = (round + k) % m;
    b = (round - k + m) % m;
  }
  if (a > b) {
    const int t = a;
    a = b;
    b = t;
  }
}

__device__ __forceinline__ int pair_index(int pa, int pb, int l) {
  return (l < JB ? pa : pb) * JB + (l & (JB - 1));
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Rotation (c, s) that zeroes the coupling of [[app, apq], [apq, aqq]] (Golub & Van Loan
// 8.5.1): t = apq / (h +- sqrt(h^2 + apq^2)), h = (aqq - app) / 2, entries at most 1 in size.
// The angle may be approximate (the coupling left over is rounding sized); c and s are brought
// back to c^2 + s^2 = 1 by one Newton step, so that thousands of rotations do not drift.
__device__ __forceinline__ void sym_schur2(float app, float aqq, float apq, float& c, float& s) {
  const float h = 0.5f * (aqq - app);
  const float r = sqrt_ftz(fmaf(h, h, apq * apq));
  const float t = apq * rcp_approx(h + copysignf(r, h));
  c = rsqrt_approx(fmaf(t, t, 1.f));
  s = t * c;
  const float e = 0.5f * fmaf(-s, s, fmaf(-c, c, 1.f));
  c = fmaf(c, e, c);
  s = fmaf(s, e, s);
}

constexpr int kInnerThreads = 512;
// Shared memory that a CTA of the inner kernel asks for beyond its own 32 KB: half an SM's, so that
// two of them never share one. They are placed while the launch before drains, onto whichever SMs
// come free, and two on an SM take turns: 15 to 34 us a round, as it happened (n = 1500).
constexpr size_t kInnerAlone = 84 * 1024;

// The tournament as a fixed permutation of positions (Brent & Luk): pair k sits at positions
// 2k, 2k + 1; after a round the player at position i moves to round_move(i), position 0 stays,
// and after 63 rounds everyone is back.
// CROSS: the pairs with one index in either block only. Those of the first block stay at the
// even positions, those of the second move on by one pair; 32 rounds.
template <bool CROSS>
__device__ __forceinline__ int round_move(int i) {
  if (CROSS) return i & 1 ? (i + 2) % JP : i;
  if (i & 1) return i == 1 ? 2 : i - 2;
  return i == 0 ? 0 : i == JP - 2 ? JP - 1 : i + 2;
}
// Column position -> offset in a stored row: even positions, then odd ones, so that the 32
// pairs of a row are 32 consecutive words of either half, before and after the move.
__device__ __forceinline__ int col_slot(int pos) { return (pos & 1) * (JP / 2) + (pos >> 1); }

// One CTA per pair of blocks: S = A[idx, idx] (64 x 64, scaled to entries at most 1), rotated
// by cyclic parallel Jacobi (32 disjoint rotations per round, 63 rounds per sweep, 32 for the
// couplings between the blocks only, which CROSS takes) until a
// sweep leaves no coupling above 1e-5 of its pivots or `inner_sweeps` sweeps ran; U (64 x 64,
// row-major) accumulates the rotations.
//
// A serial chain of rounds, so a round is built to be short: lane b of every warp computes the
// rotation of pair b for itself (three loads, three special functions), which spares an
// exchange through shared memory and its barrier; S is read from one copy and written to the
// other, already moved to the next round's positions, so that addresses are constants of the
// thread, accesses free of bank conflicts, and one barrier closes the round; U stays in
// registers, four rows a warp, a lane's two columns moving to its neighbours by shuffles.
// Bound by the latency of a round (load, rotation, update, barrier) and the 496 cycles of
// shared-memory wavefronts and shuffles in it. A sweep takes 30 us; with one warp computing
// the rotations by IEEE divisions and roots and two barriers a round it was 77 us.
template <bool CROSS>
__global__ void __launch_bounds__(kInnerThreads)
    jacobi_inner_kernel(const float* __restrict__ A, int64_t lda, int nblk, int round,
                        int inner_sweeps, float* __restrict__ Uout) {
  after_previous();
  __shared__ float ism[2 * JP * JP];  // two copies of S
  __shared__ unsigned s_max;
  constexpr int N = JP * JP;
  int pa, pb;
  rr_pair(nblk, round, blockIdx.x, pa, pb);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_max = 0;
  __syncthreads();
  float v[N / kInnerThreads];
  unsigned m = 0;  // bit patterns of non-negative floats order as they do (NaN above all)
#pragma unroll
  for (int e = 0; e < N / kInnerThreads; ++e) {
    const int idx = tid + kInnerThreads * e, i = idx / JP, j = idx % JP;
    v[e] = A[(int64_t)pair_index(pa, pb, i) * lda + pair_index(pa, pb, j)];
    m = max(m, __float_as_uint(fabsf(v[e])));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) atomicMax(&s_max, m);
  __syncthreads();
  // a power of two near the largest entry; all zero: nothing to rotate
  const bool zero = s_max == 0;
  const int ex = min(max(254 - (int)(s_max >> 23), 1), 254);
  const float scale = __uint_as_float((unsigned)ex << 23);
#pragma unroll
  for (int e = 0; e < N / kInnerThreads; ++e) {
    const int idx = tid + kInnerThreads * e, i = idx / JP, j = idx % JP;
    // index l at position l, CROSS: 2 l, or 2 (l - 32) + 1 in the second block
    if (CROSS) ism[(2 * (i & (JB - 1)) + i / JB) * JP + j] = v[e] * scale;
    else ism[i * JP + col_slot(j)] = v[e] * scale;
  }
  __syncthreads();
  // the rotation of pair `lane`, the blocks (warp, lane), (warp + 16, lane) of S, and columns
  // 2 lane, 2 lane + 1 of rows 4 warp .. of U
  const int dg = 2 * lane * JP + lane;
  const int ct = col_slot(round_move<CROSS>(2 * lane));
  const int cb = col_slot(round_move<CROSS>(2 * lane + 1));
  const int it = CROSS ? lane : 2 * lane, ib = CROSS ? JB + lane : 2 * lane + 1;
  float ut[4], ub[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    ut[u] = 4 * warp + u == it ? 1.f : 0.f;
    ub[u] = 4 * warp + u == ib ? 1.f : 0.f;
  }
  // couplings below this are already zero at float32 resolution of the pair's matrix
  float dmax = fmaxf(fabsf(ism[dg]), fabsf(ism[dg + JP + JP / 2]));
  dmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(dmax)));
  const float tiny = 1e-9f * dmax;
  int cur = 0;
  for (int sw = 0; sw < (zero ? 0 : inner_sweeps); ++sw) {
    int rotated = 0;  // the same in every warp
#pragma unroll 1
    for (int r = 0; r < (CROSS ? JB : JP - 1); ++r) {
      const float* Sc = ism + cur * N;
      float* Sn = ism + (cur ^ 1) * N;
      const float app = Sc[dg], apq = Sc[dg + JP / 2], aqq = Sc[dg + JP + JP / 2];
      float m4[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float* p = Sc + 2 * (warp + 16 * h) * JP + lane;
        m4[h][0] = p[0];
        m4[h][1] = p[JP / 2];
        m4[h][2] = p[JP];
        m4[h][3] = p[JP + JP / 2];
      }
      const float pp = fabsf(app * aqq), a2 = apq * apq;
      float c = 1.f, sn = 0.f;
      if (fabsf(apq) > tiny && a2 > 1e-14f * pp) {
        sym_schur2(app, aqq, apq, c, sn);
        // another sweep is needed while some coupling is still above 1e-5 of its pivots
        // (the smaller ones are rotated too, but leave the rest to the outer sweeps and
        // the refinement)
        if (a2 > 1e-10f * pp) rotated = 1;
      }
      // S <- J^T S J
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int a = warp + 16 * h;
        const float ca = __shfl_sync(0xffffffffu, c, a), sa = __shfl_sync(0xffffffffu, sn, a);
        // columns: (x, y) -> (c x - s y, s x + c y)
        const float n00 = c * m4[h][0] - sn * m4[h][1], n01 = sn * m4[h][0] + c * m4[h][1];
        const float n10 = c * m4[h][2] - sn * m4[h][3], n11 = sn * m4[h][2] + c * m4[h][3];
        // rows
        float o01 = ca * n01 - sa * n11, o10 = sa * n00 + ca * n10;
        if (a == lane && sa != 0.f) {
          o01 = 0.f;
          o10 = 0.f;
        }
        float* rt = Sn + round_move<CROSS>(2 * a) * JP;
        float* rb = Sn + round_move<CROSS>(2 * a + 1) * JP;
        rt[ct] = ca * n00 - sa * n10;
        rt[cb] = o01;
        rb[ct] = o10;
        rb[cb] = sa * n01 + ca * n11;
      }
      // U <- U J, then each column to the lane of its next position (round_move)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float x = c * ut[u] - sn * ub[u], y = sn * ut[u] + c * ub[u];
        if (CROSS) {
          ut[u] = x;
          ub[u] = __shfl_sync(0xffffffffu, y, (lane + JB - 1) & (JB - 1));
          continue;
        }
        const float t = __shfl_up_sync(0xffffffffu, lane == 0 ? y : x, 1);
        const float w = __shfl_down_sync(0xffffffffu, y, 1);
        ut[u] = lane == 0 ? x : t;
        ub[u] = lane == 31 ? x : w;
      }
      cur ^= 1;
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
  float* u = Uout + (int64_t)blockIdx.x * N;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float* row = u + (4 * warp + e) * JP;
    if (CROSS) {
      row[it] = ut[e];
      row[ib] = ub[e];
    } else {
      *reinterpret_cast<float2*>(row + it) = make_float2(ut[e], ub[e]);
    }
  }
}

constexpr int JPV = JP + 4;  // pitch of rows read as 16-byte words
constexpr size_t kApplySmem = 3 * (size_t)JP * JPV * sizeof(float);

// acc += X Y of 64 x 64 matrices in shared memory, thread (ty, tx): rows 4 ty + u, columns
// 4 tx + v. TX: X is stored transposed.
template <bool TX>
__device__ __forceinline__ void mm64(float (&acc)[4][4], const float (*X)[JPV],
                                     const float (*Y)[JPV], int ty, int tx) {
#pragma unroll 4
  for (int k = 0; k < JP; k += 4) {
    float a[4][4];  // [u][k]
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 v = *reinterpret_cast<const float4*>(TX ? &X[k + e][4 * ty] : &X[4 * ty + e][k]);
      if (TX) {
        a[0][e] = v.x; a[1][e] = v.y; a[2][e] = v.z; a[3][e] = v.w;
      } else {
        a[e][0] = v.x; a[e][1] = v.y; a[e][2] = v.z; a[e][3] = v.w;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 b = *reinterpret_cast<const float4*>(&Y[k + e][4 * tx]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc[u][0] = fmaf(a[u][e], b.x, acc[u][0]);
        acc[u][1] = fmaf(a[u][e], b.y, acc[u][1]);
        acc[u][2] = fmaf(a[u][e], b.z, acc[u][2]);
        acc[u][3] = fmaf(a[u][e], b.w, acc[u][3]);
      }
    }
  }
}

// blockIdx.y < pairs: A[rows_i, cols_j] <- U_i^T A[rows_i, cols_j] U_j for the pair tile
// (i, j) = (blockIdx.y, blockIdx.x); else V[rows, cols_j] <- V[rows, cols_j] U_j for 64
// consecutive rows. Both only wait for the rotations, so one launch takes them.
__global__ void __launch_bounds__(256)
    jacobi_apply_kernel(float* __restrict__ A, float* __restrict__ V, int64_t ld, int nblk,
                        int round, const float* __restrict__ Uall) {
  after_previous();
  extern __shared__ __align__(16) float asm_[];
  float(*T)[JPV] = reinterpret_cast<float(*)[JPV]>(asm_);
  float(*Uj)[JPV] = T + JP;
  float(*Ui)[JPV] = T + 2 * JP;
  const int pairs = gridDim.x;
  const bool vec = (int)blockIdx.y >= pairs;
  int ia = 0, ib = 0, ja, jb;
  rr_pair(nblk, round, blockIdx.x, ja, jb);
  if (!vec) rr_pair(nblk, round, blockIdx.y, ia, ib);
  const int64_t r0 = vec ? (int64_t)(blockIdx.y - pairs) * JP : 0;
  float* M = vec ? V : A;
  const float* ui = Uall + (int64_t)blockIdx.y * JP * JP;
  const float* uj = Uall + (int64_t)blockIdx.x * JP * JP;
  const int tid = threadIdx.x;
  auto row_of = [&](int r) { return vec ? r0 + r : (int64_t)pair_index(ia, ib, r); };
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int idx = tid + 256 * it, r = idx >> 4, c = (idx & 15) * 4;
    *reinterpret_cast<float4*>(&T[r][c]) =
        *reinterpret_cast<const float4*>(M + row_of(r) * ld + pair_index(ja, jb, c));
    *reinterpret_cast<float4*>(&Uj[r][c]) = *reinterpret_cast<const float4*>(uj + 4 * idx);
    if (!vec) *reinterpret_cast<float4*>(&Ui[r][c]) = *reinterpret_cast<const float4*>(ui + 4 * idx);
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  float acc[4][4] = {};
  mm64<false>(acc, T, Uj, ty, tx);  // T U_j
  if (!vec) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u)
      *reinterpret_cast<float4*>(&T[4 * ty + u][4 * tx]) =
          make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
    mm64<true>(acc, Ui, T, ty, tx);  // U_i^T (T U_j)
  }
  // the pair's own tile keeps what the inner sweeps left of its couplings (they need not
  // have run to convergence): the outer sweeps and the off-diagonal norm see them
#pragma unroll
  for (int u = 0; u < 4; ++u)
    *reinterpret_cast<float4*>(M + row_of(4 * ty + u) * ld + pair_index(ja, jb, 4 * tx)) =
        make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
}

// A_work = A + shift I (padded with zeros to npad), V = I.
__global__ void eigh_init_kernel(const float* __restrict__ A, int64_t n, double shift,
                                 float* __restrict__ W, float* __restrict__ V, int64_t npad) {
  const int64_t total = npad * npad;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / npad, j = idx - i * npad;
    float a = 0.f;
    if (i < n && j < n) a = (i == j) ? (float)((double)A[i * n + j] + shift) : A[i * n + j];
    W[idx] = a;
    V[idx] = (i == j) ? 1.f : 0.f;
  }
}

// norms[0] += sum of squares off the diagonal, norms[1] += on it (FP64).
__global__ void offnorm_kernel(const float* __restrict__ W, int64_t npad, double* norms) {
  double off = 0.0, on = 0.0;
  const int64_t total = npad * npad;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / npad, j = idx - i * npad;
    const double v = W[idx];
    if (i == j) on += v * v;
    else off += v * v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    off += __shfl_xor_sync(0xffffffffu, off, o);
    on += __shfl_xor_sync(0xffffffffu, on, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&norms[0], off);
    atomicAdd(&norms[1], on);
  }
}

__global__ void eigh_extract_kernel(const float* __restrict__ W, const float* __restrict__ V,
                                    int64_t npad, int64_t n, float* __restrict__ evals,
                                    float* __restrict__ evecs) {
  const int64_t total = n * n;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n, j = idx - i * n;
    evecs[idx] = V[i * npad + j];
    if (i == j) evals[i] = W[i * npad + i];
  }
}

// Spectral weights of predict.py:1277-1294 and the ensemble's covariance terms
// (predict.py:860-1005), pos = max(lambda, 0), t already scaled by the learning rate:
//   0 expm1(-pos t / N)            1 expm1(-pos t / N) / |lambda|
//   2 pos exp(-2 pos t / N)        3 exp(-pos t / N)
//   4 -expm1(-2 pos t / N) / |lambda|
//   5 -expm1(-pos t / N)           6 -expm1(-pos t / N) / |lambda|
__device__ __forceinline__ double spectral_weight(int kind, double lam, double t, double inv_norm) {
  const double pos = lam > 0.0 ? lam : 0.0;
  const double x = pos * t * inv_norm;
  switch (kind) {
    case 0: return expm1(-x);
    case 1: return expm1(-x) / fabs(lam);
    case 2: return pos * exp(-2.0 * x);
    case 3: return exp(-x);
    case 4: return -expm1(-2.0 * x) / fabs(lam);
    case 5: return -expm1(-x);
    default: return -expm1(-x) / fabs(lam);
  }
}

// out[i, t, c] = w_kind(lambda_i, t) x[i, c] for x [n, m] and times t [nt].
__global__ void spectral_scale_kernel(const float* __restrict__ evals, const double* __restrict__ ts,
                                      int64_t nt, int kind, double inv_norm,
                                      const float* __restrict__ x, int64_t n, int64_t m,
                                      float* __restrict__ out) {
  const int64_t total = n * nt * m;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = idx % m;
    const int64_t t = (idx / m) % nt;
    const int64_t i = idx / (m * nt);
    out[idx] = (float)(spectral_weight(kind, (double)evals[i], ts[t], inv_norm) *
                       (double)x[i * m + c]);
  }
}

// ---------------------------------------------------------------------------
// Refinement of the Jacobi eigenpairs (Ogita & Aishima, "Iterative refinement for
// symmetric eigenvalue decomposition", Japan J. Indust. Appl. Math. 35 (2018)):
// with X the approximate eigenvectors, R = I - X^T X and S = X^T (A X) formed in
// double-float, lambda_i = S_ii / (1 - R_ii) and X <- X + X E with
// E_ij = (S_ij + lambda_j R_ij) / (lambda_j - lambda_i) for separated pairs,
// E_ij = R_ij / 2 for pairs whose gap is not large against that numerator or is
// below 1e-6 of the largest |lambda| (a cluster: only orthogonalised), E_ii = R_ii / 2.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void df_fma_e(float a, float xh, float xl, float& sh, float& sl) {
  const float ph = a * xh;
  float pl = fmaf(a, xh, -ph);
  pl = fmaf(a, xl, pl);
  const float s2 = sh + ph;
  const float bv = s2 - sh;
  const float e = (sh - (s2 - bv)) + (ph - bv);
  sl += e + pl;
  sh = s2;
}

// C[i, j] = sum_k P[k, i] (Qh[k, j] + Ql[k, j]) + shift (Qh[i, j] + Ql[i, j]) over T x T
// tiles (T / 16 outputs per thread and side), double-float sums; P, Qh, Ql [n, n] row-major
// (Ql may be NULL). Output as FP64 (c64) or as a double-float pair (ch, cl). Bound by the FP32
// pipe (11 operations a product), so T = 32 where 64 would leave SMs without a tile.
template <int T>
__global__ void __launch_bounds__(256)
    df_gemm_tn_kernel(const float* __restrict__ P, const float* __restrict__ Qh,
                      const float* __restrict__ Ql, int64_t n, double shift,
                      double* __restrict__ c64, float* __restrict__ ch, float* __restrict__ cl) {
  constexpr int R = T / 16;
  __shared__ float Ps[16][T + 1];
  __shared__ float Hs[16][T + 1];
  __shared__ float Ls[16][T + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t i0 = (int64_t)blockIdx.y * T, j0 = (int64_t)blockIdx.x * T;
  float sh[R][R] = {}, sl[R][R] = {};
  for (int64_t k0 = 0; k0 < n; k0 += 16) {
    for (int idx = threadIdx.x; idx < 16 * T; idx += 256) {
      const int kk = idx / T, c = idx % T;
      const bool kin = k0 + kk < n;
      Ps[kk][c] = (kin && i0 + c < n) ? P[(k0 + kk) * n + i0 + c] : 0.f;
      Hs[kk][c] = (kin && j0 + c < n) ? Qh[(k0 + kk) * n + j0 + c] : 0.f;
      Ls[kk][c] = (Ql && kin && j0 + c < n) ? Ql[(k0 + kk) * n + j0 + c] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float av[R], hv[R], lv[R];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        av[u] = Ps[k][ty * R + u];
        hv[u] = Hs[k][tx * R + u];
        lv[u] = Ls[k][tx * R + u];
      }
#pragma unroll
      for (int u = 0; u < R; ++u)
#pragma unroll
        for (int v = 0; v < R; ++v) df_fma_e(av[u], hv[v], lv[v], sh[u][v], sl[u][v]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int64_t i = i0 + ty * R + u;
    if (i >= n) continue;
#pragma unroll
    for (int v = 0; v < R; ++v) {
      const int64_t j = j0 + tx * R + v;
      if (j >= n) continue;
      double val = (double)sh[u][v] + (double)sl[u][v];
      if (shift != 0.0)
        val += shift * ((double)Qh[i * n + j] + (Ql ? (double)Ql[i * n + j] : 0.0));
      if (c64) c64[i * n + j] = val;
      if (ch) {
        const float h = (float)val;
        ch[i * n + j] = h;
        cl[i * n + j] = (float)(val - (double)h);
      }
    }
  }
}

void df_gemm_tn(cudaStream_t s, const float* P, const float* Qh, const float* Ql, int64_t n,
                double shift, double* c64, float* ch, float* cl) {
  if (ceil_div(n, 64) * ceil_div(n, 64) >= 2 * 152) {
    const dim3 g((unsigned)ceil_div(n, 64), (unsigned)ceil_div(n, 64));
    df_gemm_tn_kernel<64><<<g, 256, 0, s>>>(P, Qh, Ql, n, shift, c64, ch, cl);
  } else {
    const dim3 g((unsigned)ceil_div(n, 32), (unsigned)ceil_div(n, 32));
    df_gemm_tn_kernel<32><<<g, 256, 0, s>>>(P, Qh, Ql, n, shift, c64, ch, cl);
  }
}

// R <- I - R
__global__ void identity_minus_kernel(double* __restrict__ R, int64_t n) {
  const int64_t total = n * n;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n, j = idx - i * n;
    R[idx] = (i == j ? 1.0 : 0.0) - R[idx];
  }
}

// lam_i = S_ii / (1 - R_ii); lam[n] receives max |lam_i| (zeroed by the caller).
__global__ void refine_lambda_kernel(const double* __restrict__ S, const double* __restrict__ R,
                                     int64_t n, double* __restrict__ lam) {
  double mx = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    lam[i] = S[i * n + i] / (1.0 - R[i * n + i]);
    mx = fmax(mx, fabs(lam[i]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(lam + n),
              (unsigned long long)__double_as_longlong(mx));
}

// E = the correction of X (see above); X1 = X (for the accumulate of X + X E).
__global__ void refine_e_kernel(const double* __restrict__ S, const double* __restrict__ R,
                                const double* __restrict__ lam, int64_t n, double sep,
                                float* __restrict__ E) {
  const int64_t total = n * n;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n, j = idx - i * n;
    const double r = R[idx];
    double e = 0.5 * r;
    if (i != j) {
      // separated: the gap is `sep` times the coupling or more (what a correction leaves over
      // is its square) and above the resolution of the float32 eigenvalues (1e-6 of the
      // largest); closer pairs are a cluster. By the larger of (i, j)'s and (j, i)'s coupling,
      // so that both are taken alike: half a rotation would leave the pair 1 / sep from
      // orthogonal.
      const double num = S[idx] + lam[j] * r;
      const double other = S[j * n + i] + lam[i] * R[j * n + i];
      const double gap = lam[j] - lam[i];
      if (fabs(gap) > sep * fmax(fabs(num), fabs(other)) && fabs(gap) > 1e-6 * lam[n])
        e = num / gap;
    }
    E[idx] = (float)e;
  }
}

__global__ void lam_to_float_kernel(const double* __restrict__ lam, int64_t n,
                                    float* __restrict__ evals) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    evals[i] = (float)lam[i];
}

int egrid(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g > 152 * 16 ? 152 * 16 : (g < 1 ? 1 : g));
}

struct EighWs {
  float* w;
  float* v;
  float* u;
  double* norms;
};

EighWs eigh_ws(void* ws, int64_t npad) {
  char* p = static_cast<char*>(ws);
  p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 255) & ~(uintptr_t)255);
  EighWs e;
  e.w = reinterpret_cast<float*>(p);
  e.v = e.w + npad * npad;
  e.u = e.v + npad * npad;
  const int64_t npairs = npad / JP;
  e.norms = reinterpret_cast<double*>(e.u + npairs * JP * JP);
  return e;
}

}  // namespace
}  // namespace ntg

using namespace ntg;

// Refinement buffers after the Jacobi ones: S, R [n n] f64, lam [n] f64, Yh, Yl, E [n n] f32.
size_t refine_bytes(int64_t n) {
  return (size_t)(2 * n * n + n + 1) * sizeof(double) + (size_t)3 * n * n * sizeof(float) + 1024;
}

extern "C" size_t ntg_eigh_workspace_bytes(int64_t n) {
  if (n <= 0 || n > 32768) return SIZE_MAX;
  const int64_t npad = (n + JP - 1) / JP * JP;
  return (size_t)(2 * npad * npad + (npad / JP) * JP * JP) * sizeof(float) + 2 * sizeof(double) +
         512 + refine_bytes(n);
}

extern "C" int ntg_eigh(void* stream, const float* A, int64_t n, double shift, float* evals,
                        float* evecs, int32_t max_sweeps, double tol, int32_t refine_steps,
                        void* workspace, size_t workspace_bytes, int32_t* sweeps_out) {
  NTG_REQUIRE(A && evals && evecs && workspace, "ntg_eigh: null pointer");
  NTG_REQUIRE(n > 0 && n <= 32768, "ntg_eigh: n must be in [1, 32768]");
  NTG_REQUIRE(max_sweeps > 0 && max_sweeps <= 100, "ntg_eigh: max_sweeps in [1, 100]");
  NTG_REQUIRE(refine_steps >= 0 && refine_steps <= 4, "ntg_eigh: refine_steps in [0, 4]");
  NTG_REQUIRE(workspace_bytes >= ntg_eigh_workspace_bytes(n),
              "ntg_eigh: workspace smaller than ntg_eigh_workspace_bytes(n)");
  cudaStream_t s = as_stream(stream);
  const int64_t npad = (n + JP - 1) / JP * JP;
  const int nblk = (int)(npad / JB);  // even
  const int npairs = nblk / 2;
  const EighWs e = eigh_ws(workspace, npad);
  const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if (cudaFuncSetAttribute(jacobi_apply_kernel, smem, (int)kApplySmem) != cudaSuccess ||
      cudaFuncSetAttribute(jacobi_inner_kernel<false>, smem, (int)kInnerAlone) != cudaSuccess ||
      cudaFuncSetAttribute(jacobi_inner_kernel<true>, smem, (int)kInnerAlone) != cudaSuccess)
    return check_launch("ntg_eigh");
  eigh_init_kernel<<<egrid(npad * npad), 256, 0, s>>>(A, n, shift, e.w, e.v, npad);
  note_launch();
  int sweeps = 0;
  double off2 = INFINITY;
  for (int sw = 0; sw < max_sweeps; ++sw) {
    for (int r = 0; r < nblk - 1; ++r) {
      // one inner sweep per pair and round: an inner problem driven further is undone by the
      // next rounds. A single pair is the whole matrix: to convergence. The couplings inside a
      // block are rotated in the first round of a sweep only, which pairs every block once.
      // n = 500, eigenpairs alone: 4.5 ms in ten sweeps, which an inner sweep over all couplings
      // in each round, or two, needs as well.
      launch_next_smem(s, r == 0 ? jacobi_inner_kernel<false> : jacobi_inner_kernel<true>,
                       dim3(npairs), kInnerThreads, kInnerAlone, e.w, npad, nblk, r,
                       npairs == 1 ? 8 : 1, e.u);
      launch_next_smem(s, jacobi_apply_kernel, dim3(npairs, (unsigned)(npairs + npad / JP)), 256,
                       kApplySmem, e.w, e.v, npad, nblk, r, e.u);
    }
    ++sweeps;
    if (cudaMemsetAsync(e.norms, 0, 2 * sizeof(double), s) != cudaSuccess)
      return check_launch("ntg_eigh");
    offnorm_kernel<<<egrid(npad * npad), 256, 0, s>>>(e.w, npad, e.norms);
    note_launch();
    double nh[2] = {0.0, 0.0};
    if (cudaMemcpyAsync(nh, e.norms, sizeof(nh), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return check_launch("ntg_eigh norms");
    const double fro2 = nh[0] + nh[1];
    // converged, or down at what float32 rounding leaves (sweeps converge quadratically)
    if (nh[0] <= tol * tol * fro2 || (nh[0] <= 1e-10 * fro2 && nh[0] > 0.1 * off2)) break;
    off2 = nh[0];
  }
  eigh_extract_kernel<<<egrid(n * n), 256, 0, s>>>(e.w, e.v, npad, n, evals, evecs);
  note_launch();
  if (refine_steps > 0) {
    char* rp = reinterpret_cast<char*>(
        (reinterpret_cast<uintptr_t>(e.norms + 2) + 255) & ~(uintptr_t)255);
    double* S = reinterpret_cast<double*>(rp);
    double* R = S + n * n;
    double* lam = R + n * n;
    float* yh = reinterpret_cast<float*>(lam + n + 1);
    float* yl = yh + n * n;
    float* E = yl + n * n;
    for (int it = 0; it < refine_steps; ++it) {
      // Y = (K + shift I) X (K symmetric: K^T X), S = X^T Y, R = X^T X (as -R + I below)
      df_gemm_tn(s, A, evecs, nullptr, n, shift, nullptr, yh, yl);
      df_gemm_tn(s, evecs, yh, yl, n, 0.0, S, nullptr, nullptr);
      df_gemm_tn(s, evecs, evecs, nullptr, n, 0.0, R, nullptr, nullptr);
      identity_minus_kernel<<<egrid(n * n), 256, 0, s>>>(R, n);
      if (cudaMemsetAsync(lam + n, 0, sizeof(double), s) != cudaSuccess)
        return check_launch("ntg_eigh refine");
      refine_lambda_kernel<<<egrid(n), 256, 0, s>>>(S, R, n, lam);
      // corrections up to 1e-2 where another step cleans up after them, 1e-3 in the last
      const double sep = it + 1 < refine_steps ? 1e2 : 1e3;
      refine_e_kernel<<<egrid(n * n), 256, 0, s>>>(S, R, lam, n, sep, E);
      note_launch(6);
      // X <- X + X E (the product reads a copy of X)
      if (cudaMemcpyAsync(yh, evecs, sizeof(float) * n * n, cudaMemcpyDeviceToDevice, s) !=
          cudaSuccess)
        return check_launch("ntg_eigh refine copy");
      const int rc = ntg_gemm(stream, yh, E, evecs, n, n, n, 1);
      if (rc) return rc;
    }
    lam_to_float_kernel<<<egrid(n), 256, 0, s>>>(lam, n, evals);
    note_launch();
  }
  if (sweeps_out) *sweeps_out = sweeps;
  return check_launch("ntg_eigh");
}

extern "C" int ntg_spectral_scale(void* stream, const float* evals, const double* ts, int64_t nt,
                                  int32_t kind, double norm, const float* x, int64_t n, int64_t m,
                                  float* out) {
  NTG_REQUIRE(evals && ts && x && out, "ntg_spectral_scale: null pointer");
  NTG_REQUIRE(n > 0 && m > 0 && nt > 0 && norm > 0.0, "ntg_spectral_scale: bad sizes");
  NTG_REQUIRE(kind >= 0 && kind <= 6, "ntg_spectral_scale: kind must be in [0, 6]");
  spectral_scale_kernel<<<egrid(n * nt * m), 256, 0, as_stream(stream)>>>(
      evals, ts, nt, kind, 1.0 / norm, x, n, m, out);
  note_launch();
  return check_launch("ntg_spectral_scale");
}
