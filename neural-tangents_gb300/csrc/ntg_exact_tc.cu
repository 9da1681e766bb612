// Residuals b - (A + lambda I) x of many right-hand sides with the products on the sm_103a
// tensor cores and exact sums (the slicing of Ozaki, Ogita, Oishi & Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix multiplication
// and its applications", Numer. Algorithms 59 (2012)).
//
// The products of the diagonal, (A_ii + lambda) x_i, are taken in FP64: a ridge small beside A_ii
// keeps its bits. For the others A' = A D and X' = D^-1 X, D = 2^-s with 2^2s near the diagonal,
// so that rows and columns of different scale weigh alike (|a_ij| <= sqrt(a_ii a_jj)). A row of A'
// (a column of X') is scaled by a power of two and written in balanced base-256 digits,
// |d| <= 128, which bf16 holds exactly: A' = 2^(E_i - 7) sum_p 2^-8p a_p, X' likewise with F_j,
// six digits each (48 bits below the largest entry, so float32 entries down to 2^-23 of it are
// exact). The products a_p x_q with p + q <= 5 are tcgen05.mma kind::f16, those of one level
// p + q summed in one FP32 accumulator in tensor memory: at most six products of at most 2^14
// per k, so 160 k stay below 2^24 and every sum is an exact integer. Every 160 k the six
// accumulators are drained: levels 0 - 2 into a 64-bit integer per entry, levels 3 - 5, the last
// 24 of 48 bits, into a float. What is dropped or rounded is near 2^-48 of the largest entry of
// the row of A' times that of the column of X': no more than the double-float sums lose (44 bits,
// 11 FP32 operations a product) that smaller problems take. Fewer digits do: with four and five
// small entries beside large ones cost a solution 1.6e-6 at a condition of 2.5e4; with five for A,
// its diagonal among them and no D, scales that span 1e5 cost 1e-6, and kernels that decay to
// nothing 2e-10 instead of 1e-12 after two steps.
//
// One CTA per 128 x 64 tile: TMA brings the twelve digit tiles of 32 k into a 3-stage ring
// (72 KB a stage), one thread issues the 21 x 2 MMAs of a stage, eight warps drain. Every
// wait is bounded: one that runs out raises the device error word, lets the copies and MMAs
// in flight land, frees the tensor memory and returns. Bound by the MMAs and the drain that
// follows each 160 k of them: 4096 x 4096 times 4096 x 4096 takes 3.4 ms (0.84 PFLOP/s of
// digit products) and 0.3 ms for the digits, against 24.4 ms in double-floats.
#include <cuda_bf16.h>

#include <mutex>
#include <string>

#include "ntg_exact_tc.cuh"
#include "ntg_tc.cuh"

namespace ntg {
namespace {

constexpr int XM = 128, XN = 64, XK = 32;
constexpr int PA = 6, PX = 6, LV = 6;   // digits of A, of X; levels
constexpr int XSTAGES = 3, XCHUNK = 5;  // ring stages; stages per drain (160 k)
constexpr int XA = XM * XK * 2, XB = XN * XK * 2;  // bytes of a digit tile
constexpr int XSTAGE = PA * XA + PX * XB;
constexpr int XSMEM = XSTAGES * XSTAGE + 1024 + 256;
constexpr int XTHREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 drain 32 columns each
constexpr uint32_t XTMEM = 512;
constexpr uint64_t XWAIT = 1ull << 21;
constexpr uint32_t XIDESC = tc::idesc(1, XM, XN);  // kind::f16, bf16
constexpr int kBad = 1 << 20;      // exponent of a row or column that is not finite
constexpr int kNone = -(1 << 20);  // of one that is zero
constexpr int XP = XN + 1;         // pitch of the drained tile
static_assert(3 * XM * XP * 4 <= XSTAGES * XSTAGE, "the drained tile reuses the ring");

// The e with 2^(e - 1) <= |v| < 2^e, from the bits (no FP64 operation: they are rare and slow).
__device__ __forceinline__ int exponent_of(double v) {
  const int hi = __double2hiint(v) & 0x7fffffff;
  if (hi >= 0x7ff00000) return kBad;
  if (hi == 0 && __double2loint(v) == 0) return kNone;
  return (hi >> 20) - 1022;  // a subnormal counts as the largest
}

// v 2^(bits - e) rounded to an integer, for |v| < 2^e.
__device__ __forceinline__ long long fixed_point(double v, int e, int bits) {
  const long long raw = __double_as_longlong(v);
  const int ex = (int)((raw >> 52) & 0x7ff);
  long long m = raw & 0xfffffffffffffll;
  if (ex > 0) m |= 1ll << 52;
  const int sh = (ex > 0 ? ex : 1) - 1075 + bits - e;  // v = m 2^(sh + e - bits)
  if (sh >= 0) m <<= sh;  // m 2^sh < 2^bits
  else m = sh < -62 ? 0 : (m + (1ll << (-sh - 1))) >> -sh;
  return raw < 0 ? -m : m;
}

// v = h + l: h its first 24 bits, l the others rounded to 24, from the bits where h and l are
// normal numbers.
__device__ __forceinline__ void split_bits(double v, float& h, float& l) {
  const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff;
  const unsigned lo = __double2loint(v), sign = (unsigned)hi & 0x80000000u;
  if ((unsigned)(ex - 950) < 200u) {
    h = __uint_as_float(sign | (unsigned)(ex - 896) << 23 | (unsigned)(hi & 0xfffff) << 3 |
                        lo >> 29);
    l = __uint2float_rn(lo & 0x1fffffffu) * __uint_as_float(sign | (unsigned)(ex - 948) << 23);
  } else {
    h = (float)v;
    l = isfinite(h) ? (float)(v - (double)h) : 0.f;
  }
}

// Balanced base-256 digits of v, most significant first; |v| <= 2^(8 D - 1).
template <int D>
__device__ __forceinline__ void digits_of(long long v, int (&d)[D]) {
#pragma unroll
  for (int p = D - 1; p > 0; --p) {
    d[p] = (int)((v + 128) & 255) - 128;
    v = (v - d[p]) >> 8;
  }
  d[0] = (int)v;
}

// x 2^e by exact steps (a product below 2^-126 may round once).
__device__ __forceinline__ float times_pow2(float x, int e) {
  const int h = e / 2;
  auto pow2 = [](int k) { return __int_as_float((min(max(k, -126), 127) + 127) << 23); };
  return x * pow2(h) * pow2(e - h);
}

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(XIDESC), "r"(acc));
}

// diag[k] = A_kk + lambda, S[k] = s with 2^2s near it (0 where it is no positive number).
__global__ void __launch_bounds__(256)
    scales_kernel(const float* __restrict__ A, const double* __restrict__ lambda, int64_t n,
                  double* __restrict__ diag, int* __restrict__ S) {
  const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (k >= n) return;
  const double d = (double)__ldg(A + k * n + k) + lambda[0];
  diag[k] = d;
  const int e = exponent_of(d);
  S[k] = d > 0.0 && e != kBad ? e >> 1 : 0;
}

// Digits of rows i0 .. i0 + rows of A D without its diagonal, A [n, n] -> as [PA][rows][kpad],
// exponents rowE[rows] (a row below 2^E). One CTA per row; rows past n and k past n are zero.
__global__ void __launch_bounds__(256)
    digits_rows_kernel(const float* __restrict__ A, const int* __restrict__ S, int64_t n,
                       int64_t i0, int64_t rows, int64_t kpad, __nv_bfloat16* __restrict__ as,
                       int* __restrict__ rowE) {
  __shared__ int red[8];
  const int64_t at = blockIdx.x, i = i0 + at;
  const float* a = A + i * n;
  int e = kNone;
  if (i < n) {
    for (int64_t k = threadIdx.x; k < n; k += 256) {
      const uint32_t v = __float_as_uint(__ldg(a + k)) & 0x7fffffffu;
      if (k == i || v == 0) continue;
      // a subnormal counts as the largest
      e = max(e, v >= 0x7f800000u ? kBad : (int)(v >> 23) - 126 - __ldg(S + k));
    }
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, red[w]);
  if (threadIdx.x == 0) rowE[at] = e;
  const bool some = e != kBad && e != kNone;
  for (int64_t k = threadIdx.x; k < kpad; k += 256) {
    int d[PA] = {};
    if (some && k < n && k != i) {
      float t = scalbnf(__ldg(a + k), 7 - e - __ldg(S + k));
#pragma unroll
      for (int p = 0; p < PA; ++p) {
        const float r = rintf(t);
        d[p] = (int)r;
        t = (t - r) * 256.f;  // exact
      }
    }
#pragma unroll
    for (int p = 0; p < PA; ++p) as[(p * rows + at) * kpad + k] = __int2bfloat16_rn(d[p]);
  }
}

// colF[j] = the exponent of column j of D^-1 X, X [n, m], preset to kNone.
__global__ void __launch_bounds__(256)
    exponents_kernel(const double* __restrict__ X, const int* __restrict__ S, int64_t n, int64_t m,
                     int* __restrict__ colF) {
  const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (j >= m) return;
  const int64_t k0 = (int64_t)blockIdx.y * 64, k1 = k0 + 64 < n ? k0 + 64 : n;
  int e = kNone;
#pragma unroll 8
  for (int64_t k = k0; k < k1; ++k) e = max(e, exponent_of(X[k * m + j]) + __ldg(S + k));
  // S is far smaller than what kNone and kBad are from an exponent
  if (e > kNone / 2) atomicMax(&colF[j], e < kBad / 2 ? e : kBad);
}

// Digits of the columns of D^-1 X, X [n, m] -> xs [PX][cols][kpad] (transposed); 32 x 32 blocks.
__global__ void __launch_bounds__(256)
    digits_cols_kernel(const double* __restrict__ X, const int* __restrict__ S, int64_t n,
                       int64_t m, int64_t cols, int64_t kpad, const int* __restrict__ colF,
                       __nv_bfloat16* __restrict__ xs) {
  __shared__ long long q[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t k0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32;
  const int f = j0 + tx < m ? colF[j0 + tx] : kNone;
#pragma unroll
  for (int r = ty; r < 32; r += 8) {
    const int64_t k = k0 + r, j = j0 + tx;
    q[r][tx] = k < n && f != kNone && f != kBad
                   ? fixed_point(X[k * m + j], f - __ldg(S + k), 8 * PX - 1)
                   : 0;
  }
  __syncthreads();
#pragma unroll
  for (int r = ty; r < 32; r += 8) {
    const int64_t j = j0 + r, k = k0 + tx;
    if (j >= cols || k >= kpad) continue;
    int d[PX];
    digits_of<PX>(q[tx][r], d);
#pragma unroll
    for (int p = 0; p < PX; ++p) xs[(p * cols + j) * kpad + k] = __int2bfloat16_rn(d[p]);
  }
}

struct ExactArgs {
  int64_t n, m;                  // rows of the band, columns
  int64_t k;                     // length of the sums
  int64_t arows, xcols, ni, nj;  // digit rows of a slice, tiles
  const int *rowE, *colF;
  const double *diag, *X;  // of the band
  const float* B;
  const double* B64;
  float* R;
  double* rnorm;
  int* err;
};

__global__ void __launch_bounds__(XTHREADS, 1)
    exact_residual_kernel(const __grid_constant__ CUtensorMap ta,
                          const __grid_constant__ CUtensorMap tx, const ExactArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + XSTAGES * XSTAGE);
  // [0, S): landed; [S, 2S): free; 2S: accumulators of a chunk ready; 2S + 1: drained
  uint64_t* ready = bars + 2 * XSTAGES;
  uint64_t* drained = ready + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  __shared__ int s_fail;
  // eight tiles of rows at a time against every tile of columns, so that the CTAs of a wave
  // share what they read
  const int64_t band = 8 * g.nj, b0 = blockIdx.x / band;
  const int64_t h = g.ni - 8 * b0 < 8 ? g.ni - 8 * b0 : 8, rr = blockIdx.x - b0 * band;
  const int64_t i0 = (8 * b0 + rr % h) * XM, j0 = (rr / h) * XN;
  const int nk = (int)((g.k + XK - 1) / XK), nc = (nk + XCHUNK - 1) / XCHUNK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < XSTAGES; ++s) {
      tc::mbar_init(tc::smem_u32(&bars[s]), 1);
      tc::mbar_init(tc::smem_u32(&bars[XSTAGES + s]), 1);
    }
    tc::mbar_init(tc::smem_u32(ready), 1);
    tc::mbar_init(tc::smem_u32(drained), 8);  // one arrival per draining warp
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(tmem_slot)),
                 "r"(XTMEM));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  int issued = 0;     // stages whose copies were issued
  int committed = 0;  // chunks whose MMAs were committed to `ready`
  // levels 0 - 2 in units of level 2 (below 2^48 for n < 2^16), 3 - 5 in units of level 5
  long long hi[32];
  float lo[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) hi[j] = 0, lo[j] = 0.f;
  const int half = warp >= 6 ? 32 : 0;  // a draining warp's columns

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int kc = 0; kc < nk; ++kc) {
        const int s = kc % XSTAGES;
        if (kc >= XSTAGES)
          ok = tc::mbar_wait(tc::smem_u32(&bars[XSTAGES + s]), ((kc / XSTAGES) - 1) & 1, XWAIT);
        if (!ok) break;
        const uint32_t full = tc::smem_u32(&bars[s]);
        uint8_t* st = smem + s * XSTAGE;
        tc::mbar_expect_tx(full, XSTAGE);
#pragma unroll
        for (int p = 0; p < PA; ++p)
          tc::tma_load_2d(tc::smem_u32(st + p * XA), &ta, full, kc * XK,
                          (int32_t)(p * g.arows + i0));
#pragma unroll
        for (int q = 0; q < PX; ++q)
          tc::tma_load_2d(tc::smem_u32(st + PA * XA + q * XB), &tx, full, kc * XK,
                          (int32_t)(q * g.xcols + j0));
        issued = kc + 1;
      }
      if (!ok) {
        raise_timeout(g.err);
        s_fail = 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = true;
      for (int c = 0; c < nc && ok; ++c) {
        if (c > 0) ok = tc::mbar_wait(tc::smem_u32(drained), (c - 1) & 1, XWAIT);
        if (!ok) break;
        tc::fence_after();
        const int k1 = (c + 1) * XCHUNK < nk ? (c + 1) * XCHUNK : nk;
        for (int kc = c * XCHUNK; kc < k1; ++kc) {
          const int s = kc % XSTAGES;
          ok = tc::mbar_wait(tc::smem_u32(&bars[s]), (kc / XSTAGES) & 1, XWAIT);
          if (!ok) break;
          tc::fence_after();
          const uint32_t st = tc::smem_u32(smem + s * XSTAGE);
          const bool fresh = kc == c * XCHUNK;
#pragma unroll
          for (int kk = 0; kk < XK / 16; ++kk)
#pragma unroll
            for (int p = 0; p < PA; ++p)
#pragma unroll
              for (int q = 0; q < PX; ++q)
                if (p + q < LV)
                  mma_bf16(tmem + (uint32_t)((p + q) * XN),
                           tc::smem_desc_sw64(st + p * XA + kk * 32),
                           tc::smem_desc_sw64(st + PA * XA + q * XB + kk * 32),
                           fresh && kk == 0 && p == 0 ? 0u : 1u);
          tc::commit(tc::smem_u32(&bars[XSTAGES + s]));  // frees the stage
        }
        tc::commit(tc::smem_u32(ready));
        committed = c + 1;
      }
      if (!ok) {
        raise_timeout(g.err);
        s_fail = 1;
      }
    }
  } else {
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    bool ok = true;
    for (int c = 0; c < nc; ++c) {
      ok = tc::mbar_wait(tc::smem_u32(ready), c & 1, XWAIT);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc::fence_after();
#pragma unroll
      for (int l = 0; l < LV; ++l) {
        uint32_t v[32];
        tc::tmem_ld32(lanes + (uint32_t)(l * XN + half), v);
        // exact integers of at most 2^24
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (l < 3)
            hi[j] += (long long)__float2int_rn(__uint_as_float(v[j])) * (1 << (8 * (2 - l)));
          else
            lo[j] = fmaf(__uint_as_float(v[j]), (float)(1 << (8 * (5 - l))), lo[j]);
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_u32(drained));
    }
    if (!ok && lane == 0) {
      raise_timeout(g.err);
      s_fail = 1;
    }
  }
  tc::fence_before();
  __syncthreads();
  if (s_fail) {
    // a wait ran out: the copies still in flight (the last use of each stage) and the MMAs
    // issued (the last commit) land, both bounded, before memory is released
    if (warp == 0 && lane == 0)
      for (int kc = issued > XSTAGES ? issued - XSTAGES : 0; kc < issued; ++kc)
        tc::mbar_wait(tc::smem_u32(&bars[kc % XSTAGES]), (kc / XSTAGES) & 1, XWAIT);
    if (warp == 1 && lane == 0) {
      tc::commit(tc::smem_u32(ready));
      tc::mbar_wait(tc::smem_u32(ready), committed & 1, XWAIT);
    }
    __syncthreads();
  } else {
    // the products to shared memory as sums of three floats (24 + 24 bits of levels 0 - 2,
    // levels 3 - 5), then the residuals row by row, coalesced. b less the diagonal's product
    // and the first float cancel exactly where they cancel. One FP64 operation an entry: six,
    // with the conversions, took 12 us a tile.
    float* tile = reinterpret_cast<float*>(smem);
    if (warp >= 2) {
      const int row = (warp & 3) * 32 + lane;
      const int64_t i = i0 + row;
      const int e = i < g.n ? g.rowE[i] : kNone;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int64_t jj = j0 + half + j;
        const int f = jj < g.m ? __ldg(g.colF + jj) : kNone;
        float h1 = 0.f, h2 = 0.f, l1 = 0.f;
        if (e == kBad || f == kBad) {
          h1 = NAN;
        } else if (e != kNone && f != kNone) {
          const int sc = e + f - 14 - 16;  // of level 2
          h1 = __ll2float_rn(hi[j]);
          h2 = times_pow2(__ll2float_rn(hi[j] - __float2ll_rn(h1)), sc);
          h1 = times_pow2(h1, sc);
          l1 = times_pow2(lo[j], sc - 24);
        }
        float* t = tile + row * XP + half + j;
        t[0] = h1;
        t[XM * XP] = h2;
        t[2 * XM * XP] = l1;
      }
    }
    __syncthreads();
    float mx = 0.f;
    for (int idx = threadIdx.x; idx < XM * XN; idx += XTHREADS) {
      const int64_t i = i0 + idx / XN, j = j0 + idx % XN;
      if (i >= g.n || j >= g.m) continue;
      const int64_t at = i * g.m + j;
      const float* t = tile + (idx / XN) * XP + idx % XN;
      float dh, dl;
      split_bits(fma(-__ldg(g.diag + i), __ldg(g.X + at), g.B64 ? g.B64[at] : 0.0), dh, dl);
      const float b = g.B64 ? 0.f : g.B[at];
      const float s = __fadd_rn(b, dh), z = __fsub_rn(s, b);
      const float e = __fadd_rn(__fsub_rn(b, __fsub_rn(s, z)), __fsub_rn(dh, z));  // b + dh - s
      const float r = ((s - t[0]) + ((e + dl) - t[XM * XP])) - t[2 * XM * XP];
      g.R[at] = r;
      mx = fmaxf(mx, fabsf(r));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0 && mx > 0.f)
      atomicMax(reinterpret_cast<unsigned long long*>(g.rnorm),
                (unsigned long long)__double_as_longlong((double)mx));
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(XTMEM));
}

// A's digits, 3 times its size, are made for a band of at most 512 MiB of rows at a time (one
// tile at least; one band up to n = 6656) and X's for all columns: 12 bytes an entry where the
// double-float split takes 8.
struct ExactWs {
  int64_t kpad, arows, xcols;  // arows: of a band
  __nv_bfloat16 *as, *xs;
  int *rowE, *colF, *S;
  double* diag;
  size_t bytes;
};

ExactWs exact_ws(void* ws, int64_t n, int64_t m) {
  ExactWs w;
  w.kpad = ceil_div(n, XK) * XK;
  const int64_t fit = (1ll << 29) / (PA * w.kpad * 2) / XM * XM, pad = ceil_div(n, XM) * XM;
  w.arows = pad < fit ? pad : fit > XM ? fit : XM;
  w.xcols = ceil_div(m, XN) * XN;
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t a = up((size_t)PA * w.arows * w.kpad * 2), x = up((size_t)PX * w.xcols * w.kpad * 2);
  const size_t e = up((size_t)w.arows * 4), f = up((size_t)w.xcols * 4), d = up((size_t)n * 8);
  char* p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
  w.as = reinterpret_cast<__nv_bfloat16*>(p);
  w.xs = reinterpret_cast<__nv_bfloat16*>(p + a);
  w.rowE = reinterpret_cast<int*>(p + a + x);
  w.colF = reinterpret_cast<int*>(p + a + x + e);
  w.diag = reinterpret_cast<double*>(p + a + x + e + f);
  w.S = reinterpret_cast<int*>(p + a + x + e + f + d);
  w.bytes = a + x + e + f + d + up((size_t)n * 4) + 256;
  return w;
}

__global__ void fill_int_kernel(int* p, int64_t n, int v) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

}  // namespace

bool exact_residual_pays(int64_t n, int64_t m) { return n * n * m >= (1ll << 26); }

size_t exact_residual_bytes(int64_t n, int64_t m) { return exact_ws(nullptr, n, m).bytes; }

int exact_residual(cudaStream_t s, const float* A, int64_t n, const double* lambda, const float* B,
                   const double* B64, const double* X, int64_t m, float* R, double* rnorm,
                   void* workspace, bool same_a) {
  const ExactWs w = exact_ws(workspace, n, m);
  NTG_REQUIRE(PA * w.arows < (1ll << 31) && PX * w.xcols < (1ll << 31) && w.kpad < (1ll << 31),
              "exact residual: sizes too large");
  int* const err = device_error_word();
  NTG_REQUIRE(err, "exact residual: no device error word");
  CUtensorMap ma, mx;
  int rc = tc::make_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w.as, PA * w.arows, w.kpad,
                           w.kpad, XM, XK, "exact residual", CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  rc = tc::make_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w.xs, PX * w.xcols, w.kpad,
                       w.kpad, XN, XK, "exact residual", CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  const cudaError_t e = cudaFuncSetAttribute(
      exact_residual_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XSMEM);
  if (e != cudaSuccess) return fail(NTG_ERR_CUDA, std::string("exact residual: ") + cudaGetErrorString(e));
  if (!same_a) {
    scales_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(A, lambda, n, w.diag, w.S);
    note_launch();
  }
  fill_int_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, s>>>(w.colF, m, kNone);
  exponents_kernel<<<dim3((unsigned)ceil_div(m, 256), (unsigned)ceil_div(n, 64)), 256, 0, s>>>(
      X, w.S, n, m, w.colF);
  digits_cols_kernel<<<dim3((unsigned)ceil_div(w.kpad, 32), (unsigned)ceil_div(w.xcols, 32)), 256,
                       0, s>>>(X, w.S, n, m, w.xcols, w.kpad, w.colF, w.xs);
  note_launch(3);
  for (int64_t i0 = 0; i0 < n; i0 += w.arows) {
    if (!same_a || n > w.arows) {
      digits_rows_kernel<<<(unsigned)w.arows, 256, 0, s>>>(A, w.S, n, i0, w.arows, w.kpad, w.as,
                                                           w.rowE);
      note_launch();
    }
    const int64_t rows = n - i0 < w.arows ? n - i0 : w.arows;
    const int64_t ni = ceil_div(rows, XM), nj = w.xcols / XN;
    const ExactArgs g{rows, m, n, w.arows, w.xcols, ni, nj, w.rowE, w.colF, w.diag + i0,
                      X + i0 * m, B ? B + i0 * m : nullptr, B64 ? B64 + i0 * m : nullptr,
                      R + i0 * m, rnorm, err};
    exact_residual_kernel<<<(unsigned)(ni * nj), XTHREADS, XSMEM, s>>>(ma, mx, g);
    note_launch();
  }
  return check_launch("exact residual");
}

}  // namespace ntg
