// Batched right-hand sides against one factorisation, with a fixed number of refinement sweeps and no
// host synchronisation (a call only launches kernels on its stream, so time steps can be captured in a
// CUDA graph).  Time-stepped problems in the reference rebuild and refactor on every step
// (demos/Advection/00_advection_with_rbf.py:83-93); here the factors of updes_factor are reused and R
// right-hand sides (R <= 64) advance together:
//   X = M^-1 Bs;  repeat `sweeps` times:  X += M^-1 (Bs - Ks X)
// with Ks the equilibrated K (the exact sum of the solve workspace's double-float planes) and M^-1 the LU factors
// applied in double-float arithmetic.  updes_batch_prepare derives once per factorisation what the calls read:
//   * the inverses of the factors' 64 x 64 diagonal blocks and each block row times its inverse (or, for an ill-conditioned
//     block, as it is), as hi/lo FP32 planes: a solve leaves residuals of about 2^-48, on the FP32 pipes;
//   * the digits of Ks and of the value matrix [Phi P], without the polynomial columns, for the tensor-core products
//     (gemm_tc64.cu).
//
// A thread's double-float sums are renormalised every eight terms, so their error stays at about 2^-46 of the running sum
// however many terms it adds.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "common.cuh"
#include "gemm_tc.cuh"
#include "lu.cuh"
#include "rbf.cuh"
#include "stats.cuh"

namespace {

constexpr int kB = 64;       // block rows
constexpr int kMaxR = 64;    // right-hand sides per call
constexpr int kCG = 8;       // right-hand sides per triangular-solve CTA
constexpr int kLdt = kB + 8; // row stride of a staged tile: the 4 rows x 8 columns a warp reads at once fall in 32 banks
constexpr int kChunk = 256;  // value rows staged at a time
constexpr int kMaxM = 15;    // monomials of a system, at most (degree 4)
constexpr int kMaxBlocks = 1024;  // block rows; a factorisation has at most 800 (n <= 51,200)

__device__ __forceinline__ float2 sub2(float2 y, float2 x) { return __ffma2_rn(x, make_float2(-1.f, -1.f), y); }

// Double-float accumulators of a pair of columns: (sh, sl) += (a + al) * (b + bl), dropping al * bl; nb = -b.  Packed
// FP32x2 instructions, 12 of them: the negated product comes from the negated operand (a negation of a pair costs two
// more), and the pair is renormalised by its owner after a few terms.
__device__ __forceinline__ void df_mac2(float a, float al, float2 b, float2 nb, float2 bl, float2& sh, float2& sl) {
  const float2 a2 = make_float2(a, a), al2 = make_float2(al, al);
  const float2 np = __fmul2_rn(a2, nb);
  const float2 e = __ffma2_rn(a2, b, np);
  const float2 s = sub2(sh, np);
  const float2 bb = sub2(s, sh);
  const float2 t = sub2(sub2(sh, sub2(s, bb)), __fadd2_rn(np, bb));
  sl = __fadd2_rn(sl, __fadd2_rn(t, __ffma2_rn(a2, bl, __ffma2_rn(al2, b, e))));
  sh = s;
}

// (sh, sl) += (h, l)
__device__ __forceinline__ void df_add(float h, float l, float& sh, float& sl) {
  const float s = __fadd_rn(sh, h);
  const float bb = __fsub_rn(s, sh);
  float t = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bb)), __fsub_rn(h, bb));
  t = __fadd_rn(t, __fadd_rn(sl, l));
  sh = __fadd_rn(s, t);
  sl = __fsub_rn(t, __fsub_rn(sh, s));
}

__device__ __forceinline__ void split(double v, float& h, float& l) {
  h = float(v);
  l = float(v - double(h));
}

// Header of the batch workspace: the system and the factors that it was prepared for.  N: of n = N + M; values: the
// value matrix was prepared as well (not on local supports).
struct BatchHeader {
  int32_t n, precision, valid, generation, N, values;
};
// Whether a preparation is of the factors in the solve workspace (its state words).
__device__ __forceinline__ bool describes(const BatchHeader* hdr, const int32_t* state, int n, int N) {
  return state[0] == n && state[2] == 1 && hdr->n == n && hdr->N == N && hdr->valid == 1 && hdr->precision == state[1] &&
         hdr->generation == state[3];
}

// A solved entry on its way to the blocks after it: two words, each with a tag in its high half (set: 1) and one FP32
// half of the double-float value in its low half, each stored and loaded as one single-copy-atomic access.
struct alignas(16) Word {
  unsigned long long hi, lo;
};
__device__ __forceinline__ void put_word(Word* w, float h, float l) {
  const unsigned long long tag = 1ull << 32;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&w->hi), "l"(tag | __float_as_uint(h)) : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&w->lo), "l"(tag | __float_as_uint(l)) : "memory");
}
__device__ __forceinline__ Word get_word(const Word* w) {  // past L1, so that a second look sees new stores
  Word v;
  asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(v.hi), "=l"(v.lo) : "l"(w) : "memory");
  return v;
}
__device__ __forceinline__ bool is_set(const Word& w) { return (w.hi >> 32) == 1 && (w.lo >> 32) == 1; }

// The polynomial columns of K and of the value matrix, and their coefficients, are of another size than the kernel's, with
// which they would share a digit scale, and few: FP64 multiply-adds.  KP (n x M) and VP (N x M), written while preparing
// (from the planes and the nodes in each call they cost 20 us of a step's 4,700 at n = 6,403).
__global__ void polynomial_columns_kernel(const float* __restrict__ Khi, const float* __restrict__ Klo, int64_t ld,
                                          const double* __restrict__ nodes, int n, int N, double* __restrict__ KP,
                                          double* __restrict__ VP) {
  const int M = n - N, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * M) return;
  const int i = e / M, k = e % M;
  KP[e] = double(Khi[int64_t(i) * ld + N + k]) + double(Klo[int64_t(i) * ld + N + k]);
  if (i < N) VP[e] = monomial_terms(k, nodes[2 * i], nodes[2 * i + 1]).m;
}

// s + sum_k P[k] X[k ldx], k < M <= kMaxM, the loads in flight together
__device__ __forceinline__ double add_polynomial(double s, const double* __restrict__ P, const double* __restrict__ X,
                                                 int64_t ldx, int M) {
  double p[kMaxM], x[kMaxM];
#pragma unroll
  for (int k = 0; k < kMaxM; ++k) {
    if (k >= M) break;
    p[k] = P[k];
    x[k] = X[k * ldx];
  }
#pragma unroll
  for (int k = 0; k < kMaxM; ++k) {
    if (k >= M) break;
    s = fma(p[k], x[k], s);
  }
  return s;
}

// Res = Bs - sum_p partial[p] - KP X[N:] (partials: splits x n x 64, the product with K's first N columns)
__global__ void batch_residual_kernel(const double* __restrict__ Bs, const double* __restrict__ partial, int splits,
                                      int n, int N, int R, const double* __restrict__ KP, const double* __restrict__ X,
                                      double* __restrict__ Res, const int32_t* __restrict__ skip) {
  if (skip && *skip) return;
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= int64_t(n) * R) return;
  const int64_t i = e / R, c = e % R;
  double s = 0.0;
  for (int p = 0; p < splits; ++p) s += partial[(int64_t(p) * n + i) * kMaxR + c];
  Res[e] = Bs[e] - add_polynomial(s, KP + i * (n - N), X + int64_t(N) * R + c, R, n - N);
}

// vals[i][c] = sum_p partial[p][i][c] + sum_k VP[i][k] C[N + k][c]; NaN, and UPDES_ERR_INVALID in the status, if the header
// does not describe a preparation of this system with its values
__global__ void batch_values_kernel(const double* __restrict__ partial, int splits, int N, int n, int R,
                                    const double* __restrict__ VP, const double* __restrict__ C, int64_t ldc,
                                    double* __restrict__ vals, int64_t ldv, const int32_t* __restrict__ state,
                                    const BatchHeader* __restrict__ hdr, DeviceStatus* st) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool ok = describes(hdr, state, n, N) && hdr->values == 1;
  if (!ok && e == 0) status_error(st, UPDES_ERR_INVALID);
  if (e >= int64_t(N) * R) return;
  const int64_t i = e / R, c = e % R;
  double s = 0.0;
  for (int p = 0; p < splits; ++p) s += partial[(int64_t(p) * N + i) * kMaxR + c];
  s = add_polynomial(s, VP + i * (n - N), C + int64_t(N) * ldc + c, ldc, n - N);
  vals[i * ldv + c] = ok ? s : __longlong_as_double(0x7ff8000000000000ll);
}

// Bs[i][c] = dr_i * Q[i][c] (i < N), 0 for the polynomial rows.  The solve workspace must hold factors of
// this size and the batch header must describe them (same generation); otherwise the status records
// UPDES_ERR_INVALID and the right-hand sides become NaN, so nothing downstream passes for a solution.
__global__ void batch_rhs_kernel(const double* __restrict__ Q, int64_t ldq, int N, int n, int R,
                                 const double* __restrict__ dr, double* __restrict__ Bs,
                                 const int32_t* __restrict__ state, const BatchHeader* __restrict__ hdr,
                                 DeviceStatus* st) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool ok = describes(hdr, state, n, N);
  if (!ok && e == 0) status_error(st, UPDES_ERR_INVALID);
  if (e >= int64_t(n) * R) return;
  const int i = int(e / R), c = int(e % R);
  Bs[e] = !ok ? __longlong_as_double(0x7ff8000000000000ll) : (i < N ? dr[i] * Q[int64_t(i) * ldq + c] : 0.0);
}

// out[i][c] (ld = ldo) = dc_i * X[i][c]
__global__ void batch_unscale_kernel(const double* __restrict__ X, const double* __restrict__ dc, int n, int R,
                                     double* __restrict__ out, int64_t ldo) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= int64_t(n) * R) return;
  const int i = int(e / R), c = int(e % R);
  out[int64_t(i) * ldo + c] = dc[i] * X[e];
}

// A block row is solved with its diagonal block's inverse I_b either before or after its sum: x_b = I_b y_b + sum G x with
// G = -I_b T (a hand-off costs one product), or, where |I_b| |T_bb| has a row sum above kPremultiplied, x_b = I_b r with
// r = y_b - sum T x and one step of refinement, x_b += I_b (r - T_bb x_b) (three products more).  The first rounds
// I_b y_b and the products before they cancel, which leaves residuals of up to that row sum times 2^-48 (a substitution:
// 2^-48), and a refinement sweep brings those down only while they are small: r^7 with 576 nodes has row sums of 5e5, and
// its values were wrong by 8e-5 without a sweep, 5e-10 with one (by substitution 5e-10 and 3e-11).  Below the limit one sweep
// leaves what it leaves after a substitution (r^3, r^5, r^7 and multiquadrics of 600 to 3,000 nodes), so a solve
// on FP64 factors has at least one.  At a limit of 256 the steps of 6,403 multiquadrics took
// 10 % longer, at 4,096 0.5 %, here 0.1 %.
constexpr double kPremultiplied = 16384.0;

// Three pairs of 64 x 64 hi/lo planes a diagonal block: what the right-hand side is multiplied by (I_b, or the identity),
// and for the second form I_b and -T_bb.
constexpr int kTilePlanes = 6;

// Inverses of the diagonal blocks of a triangular factor F (LOWER: unit lower), 64 x 64 each, their planes (see above) and
// which form their rows take (after[blk] = 1: the second).  Rows and columns beyond n count as the identity.
struct InverseSmem {
  double T[kB][kB + 1], I[kB][kB + 1];
};

template <typename TF, bool LOWER>
__global__ void __launch_bounds__(256) tri_inverse_kernel(const TF* __restrict__ F, int64_t ldf, int n,
                                                          double* __restrict__ inv, float* __restrict__ tiles,
                                                          int32_t* __restrict__ after) {
  extern __shared__ double inv_smem[];
  InverseSmem& sm = *reinterpret_cast<InverseSmem*>(inv_smem);
  __shared__ double row_sum[kB];
  const int blk = blockIdx.x, r0 = blk * kB, tid = threadIdx.x;
  for (int e = tid; e < kB * kB; e += blockDim.x) {
    const int i = e >> 6, j = e & 63;
    double t = (r0 + i < n && r0 + j < n) ? double(F[int64_t(r0 + i) * ldf + r0 + j]) : (i == j ? 1.0 : 0.0);
    if (LOWER ? j >= i : j < i) t = LOWER && i == j ? 1.0 : 0.0;  // the triangle alone
    sm.T[i][j] = t;
  }
  __syncthreads();
  if (tid < kB) {  // a column of the inverse by substitution
    const int j = tid;
    for (int s = 0; s < kB; ++s) {
      const int i = LOWER ? s : kB - 1 - s;
      double x = i == j ? 1.0 : 0.0;
      if (LOWER) {
        for (int k = j; k < i; ++k) x = fma(-sm.T[i][k], sm.I[k][j], x);
      } else {
        for (int k = i + 1; k <= j; ++k) x = fma(-sm.T[i][k], sm.I[k][j], x);
        x /= sm.T[i][i];
      }
      sm.I[i][j] = x;
    }
  }
  __syncthreads();
  if (tid < kB) {
    double t = 0.0;
    for (int k = 0; k < kB; ++k) t += fabs(sm.T[tid][k]);
    row_sum[tid] = t;
  }
  __syncthreads();
  bool large = false;
  if (tid < kB) {
    double t = 0.0;
    for (int k = 0; k < kB; ++k) t = fma(fabs(sm.I[tid][k]), row_sum[k], t);  // of |I_b| |T_bb|
    large = !(t <= kPremultiplied);
  }
  const bool second = __syncthreads_or(large);
  if (tid == 0) after[blk] = second;
  float* out = tiles + int64_t(blk) * kTilePlanes * kB * kB;
  for (int e = tid; e < kB * kB; e += blockDim.x) {
    const int i = e >> 6, j = e & 63;
    const double x = sm.I[i][j];
    inv[int64_t(blk) * kB * kB + e] = x;
    split(second ? (i == j ? 1.0 : 0.0) : x, out[e], out[kB * kB + e]);
    if (!second) continue;
    split(x, out[2 * kB * kB + e], out[3 * kB * kB + e]);
    split(-sm.T[i][j], out[4 * kB * kB + e], out[5 * kB * kB + e]);
  }
}

// G = -I_b T, or -T for the rows of the second form, for every block T of block row b beside the diagonal (below it in L,
// above it in U), as hi/lo planes in the place of T; a CTA a block, the lower triangle's inverses in invL, the upper's in invU.
template <typename TF>
__global__ void __launch_bounds__(256) tri_premultiply_kernel(const TF* __restrict__ F, int64_t ldf, int n,
                                                              const double* __restrict__ invL,
                                                              const double* __restrict__ invU,
                                                              const int32_t* __restrict__ afterL,
                                                              const int32_t* __restrict__ afterU,
                                                              float* __restrict__ Gh, float* __restrict__ Gl) {
  extern __shared__ double inv_smem[];
  InverseSmem& sm = *reinterpret_cast<InverseSmem*>(inv_smem);
  const int b = blockIdx.y, q = blockIdx.x, tid = threadIdx.x;
  if (b == q) return;
  const double* inv = (q < b ? invL : invU) + int64_t(b) * kB * kB;
  const int r0 = b * kB, c0 = q * kB;
  if ((q < b ? afterL : afterU)[b]) {
    for (int e = tid; e < kB * kB; e += blockDim.x) {
      const int r = r0 + (e >> 6), c = c0 + (e & 63);
      if (r < n && c < ldf)
        split(c < n ? -double(F[int64_t(r) * ldf + c]) : 0.0, Gh[int64_t(r) * ldf + c], Gl[int64_t(r) * ldf + c]);
    }
    return;
  }
  for (int e = tid; e < kB * kB; e += blockDim.x) {
    const int i = e >> 6, j = e & 63;
    sm.I[i][j] = inv[e];
    sm.T[i][j] = (r0 + i < n && c0 + j < n) ? double(F[int64_t(r0 + i) * ldf + c0 + j]) : 0.0;
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  double acc[4][4] = {};
#pragma unroll 4
  for (int k = 0; k < kB; ++k) {
    double a[4], t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { a[u] = -sm.I[ty + 16 * u][k]; t[u] = sm.T[k][tx + 16 * u]; }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], t[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = r0 + ty + 16 * u, c = c0 + tx + 16 * v;
      if (r < n && c < ldf) split(c < n ? acc[u][v] : 0.0, Gh[int64_t(r) * ldf + c], Gl[int64_t(r) * ldf + c]);
    }
}

// ---------------------------------------------------------------------------
// Triangular solve of n x R right-hand sides (LOWER: unit lower, forward; else upper, backward).
// One CTA per (64-row block, group of 8 right-hand sides), taken in ticket order.  Block b is
//   x_b = I_b y_b + sum_q G_bq x_q,   G_bq = -I_b T_bq,
// with I_b the inverted diagonal block (or, by after[b], the second form above): what is left to do when x_{b-1} arrives is
// one 64 x 64 product and one hand-off (a substitution inside each block and hand-offs through counters and fences made the
// chain 32 us a block).
// Tiles are staged by cp.async one ahead, and the words of a block are read one tile ahead of their use, so blocks
// solved long ago cost no waiting.
// Bound by the FP32 pipes for many columns (12 packed instructions per two double-float multiply-adds, which issue every
// other cycle: 64 columns of n = 6,406 take 0.96 ms a triangle), by the chain for few (8
// columns: 0.45 ms, 4.4 us a block).
// A thread owns rows rg + 16 u (u < 4), the columns 2 cg and 2 cg + 1, and every eighth term of the inner sum.
constexpr int kTriThreads = 512, kKs = 8;
struct TriSmem {
  float F[2][2][kB][kLdt];   // [buffer][hi, lo]
  float Xn[2][kB][kCG];  // the high words negated
  float Xh[2][kB][kCG], Xl[2][kB][kCG];
};

// One (block row, column group).  The second form has code of its own, out of line: a block runs its code once, on the chain,
// and the form's instructions between those of the first cost that 0.2 us a block, taken or not.
template <bool LOWER, bool SECOND>
__device__ __noinline__ void tri_block(TriSmem& sm, int t, int cbase, const float* __restrict__ Gh,
                                          const float* __restrict__ Gl, int64_t ldg, const float* __restrict__ tiles, int n,
                                          int R, const double* __restrict__ Bin, const int32_t* __restrict__ perm,
                                          const Word* win, Word* wout, double* Y, int accumulate, DeviceStatus* st) {
  const int tid = threadIdx.x;
  const int ks = tid & (kKs - 1), rg = (tid >> 3) & 15, cg = tid >> 7;
  const int nblk = int(ceil_div(n, kB));
  const int blk = LOWER ? t : nblk - 1 - t, r0 = blk * kB;
  auto block_at = [&](int q) { return LOWER ? q : nblk - 1 - q; };  // the q-th block to be solved

  // item 0 is the inverse (or the identity) times the right-hand side, item i, 1 <= i <= t, the product with the (i-1)-th
  // solved block; items t + 1 .. t + 3 are those of the second form: I_b r, -T_bb x, I_b times what is left
  auto stage = [&](int i) {
    const float *hi, *lo;
    int64_t ld;
    int rows = kB, cols = kB;
    if (i == 0 || (SECOND && i > t)) {
      hi = tiles + (int64_t(blk) * kTilePlanes + (i == 0 ? 0 : i == t + 2 ? 4 : 2)) * kB * kB;
      lo = hi + kB * kB;
      ld = kB;
    } else {
      const int c0 = block_at(i - 1) * kB;
      hi = Gh + int64_t(r0) * ldg + c0;
      lo = Gl + int64_t(r0) * ldg + c0;
      ld = ldg;
      rows = n - r0;
      cols = n - c0;
    }
#pragma unroll
    for (int k = 0; k < 2 * kB * kB / 4 / kTriThreads; ++k) {
      const int e = tid + kTriThreads * k, p = e >> 10, row = (e >> 4) & 63, ch = (e & 15) * 4;
      const bool ok = row < rows && ch < cols;  // the planes' columns from n on are zero
      const float* src = (p ? lo : hi) + (ok ? int64_t(row) * ld + ch : 0);
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&sm.F[i & 1][p][row][ch]));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int xr = tid >> 3, xc = tid & 7;  // the entry of a 64 x 8 block that this thread brings to shared memory
  auto word_at = [&](int i) -> const Word* {
    const int row = block_at(i - 1) * kB + xr, c = cbase + xc;
    return (row < n && c < R) ? wout + int64_t(row) * R + c : nullptr;
  };
  auto fetch = [&](int i) {
    const Word* w = word_at(i);
    return w ? get_word(w) : Word{1ull << 32, 1ull << 32};
  };

  stage(0);
  Word pre{1ull << 32, 1ull << 32};  // the right-hand side's entry, then words one item ahead
  if (r0 + xr < n && cbase + xc < R) {
    if (LOWER) {
      // (a workspace may hold no factors, and then no permutation either)
      float h, l;
      split(Bin[int64_t(min(max(perm[r0 + xr], 0), n - 1)) * R + cbase + xc], h, l);
      pre = Word{(1ull << 32) | __float_as_uint(h), (1ull << 32) | __float_as_uint(l)};
    } else {
      pre = get_word(win + int64_t(r0 + xr) * R + cbase + xc);
    }
  }
  float2 ah[4], al[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) ah[u] = al[u] = make_float2(0.f, 0.f);
  // The sum over the eight threads of a row: each exchange also halves what a thread keeps, down to one row of a pair
  // of columns in two threads, so that thread ks ends with row rg + 16 (ks & 3), column 2 cg + (ks >> 2), in (h, l).
  auto reduce = [&](float& h, float& l) {
#pragma unroll
    for (int u = 0; u < 4; u += 2) {  // lanes that differ in bit 0 split rows u, u + 1
      const bool up = ks & 1;
      const float2 sh = up ? ah[u] : ah[u + 1], sl = up ? al[u] : al[u + 1];
      float2 kh = up ? ah[u + 1] : ah[u], kl = up ? al[u + 1] : al[u];
      df_add(__shfl_xor_sync(0xffffffffu, sh.x, 1), __shfl_xor_sync(0xffffffffu, sl.x, 1), kh.x, kl.x);
      df_add(__shfl_xor_sync(0xffffffffu, sh.y, 1), __shfl_xor_sync(0xffffffffu, sl.y, 1), kh.y, kl.y);
      ah[u] = kh;
      al[u] = kl;
    }
    float2 rh, rl;
    {
      const bool up = ks & 2;
      const float2 sh = up ? ah[0] : ah[2], sl = up ? al[0] : al[2];
      rh = up ? ah[2] : ah[0];
      rl = up ? al[2] : al[0];
      df_add(__shfl_xor_sync(0xffffffffu, sh.x, 2), __shfl_xor_sync(0xffffffffu, sl.x, 2), rh.x, rl.x);
      df_add(__shfl_xor_sync(0xffffffffu, sh.y, 2), __shfl_xor_sync(0xffffffffu, sl.y, 2), rh.y, rl.y);
    }
    const bool up = ks & 4;
    h = up ? rh.y : rh.x;
    l = up ? rl.y : rl.x;
    df_add(__shfl_xor_sync(0xffffffffu, up ? rh.x : rh.y, 4), __shfl_xor_sync(0xffffffffu, up ? rl.x : rl.y, 4), h, l);
  };
  // ah, al += the staged item times its 64 x 8 block
  auto multiply = [&](int b) {
#pragma unroll
    for (int k = 0; k < kB / kKs; ++k) {
      const int kk = kKs * k + ks;
      const float2 xh = *reinterpret_cast<const float2*>(&sm.Xh[b][kk][2 * cg]);
      const float2 xn = *reinterpret_cast<const float2*>(&sm.Xn[b][kk][2 * cg]);
      const float2 xl = *reinterpret_cast<const float2*>(&sm.Xl[b][kk][2 * cg]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        df_mac2(sm.F[b][0][rg + 16 * u][kk], sm.F[b][1][rg + 16 * u][kk], xh, xn, xl, ah[u], al[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // eight terms on: renormalised
      const float2 s = __fadd2_rn(ah[u], al[u]);
      al[u] = sub2(al[u], sub2(s, ah[u]));
      ah[u] = s;
    }
  };
  for (int i = 0; i <= t; ++i) {
    const int b = i & 1;
    if (i > 0) {
      long long it = 0;
      while (!is_set(pre)) {
        if (++it > spin_limit()) {
          status_error(st, UPDES_ERR_TIMEOUT);
          atomicCAS(&st->timeout_tag, 0, 30);
          break;
        }
        if (it > 64) __nanosleep(20);
        pre = get_word(word_at(i));
      }
    }
    sm.Xh[b][xr][xc] = __uint_as_float(uint32_t(pre.hi));
    sm.Xn[b][xr][xc] = -__uint_as_float(uint32_t(pre.hi));
    sm.Xl[b][xr][xc] = __uint_as_float(uint32_t(pre.lo));
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (i < t) {
      stage(i + 1);
      pre = fetch(i + 1);
    }
    multiply(b);
  }
  const int own_row = rg + 16 * (ks & 3), own_col = 2 * cg + (ks >> 2);
  float h, l;
  reduce(h, l);
  if constexpr (SECOND) {  // (h, l) is r; x = I_b r, x += I_b (r - T_bb x)
    const float rh = h, rl = l;
    float xh = 0.f, xl = 0.f;
    stage(t + 1);
    for (int i = t + 1; i <= t + 3; ++i) {
      const int b = i & 1;
      if (i == t + 2) {
        xh = h;
        xl = l;
      } else if (i == t + 3) {
        df_add(rh, rl, h, l);
      }
      sm.Xh[b][own_row][own_col] = h;
      sm.Xn[b][own_row][own_col] = -h;
      sm.Xl[b][own_row][own_col] = l;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      if (i < t + 3) stage(i + 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) ah[u] = al[u] = make_float2(0.f, 0.f);
      multiply(b);
      reduce(h, l);
    }
    df_add(xh, xl, h, l);
  }
  const int own = r0 + own_row, c = cbase + own_col;
  if (own < n && c < R) {
    const int64_t at = int64_t(own) * R + c;
    put_word(wout + at, h, l);
    if (!LOWER) {
      const double x = double(h) + double(l);
      Y[at] = accumulate ? Y[at] + x : x;
    }
  }
}

template <bool LOWER>
__global__ void __launch_bounds__(kTriThreads) batch_tri_kernel(const float* __restrict__ Gh,
                                                                const float* __restrict__ Gl, int64_t ldg,
                                                                const float* __restrict__ tiles,
                                                                const int32_t* __restrict__ after, int n, int R,
                                                                const double* __restrict__ Bin,
                                                                const int32_t* __restrict__ perm, const Word* win,
                                                                Word* wout, double* Y, int accumulate, int* ticket,
                                                                DeviceStatus* st, const int32_t* __restrict__ skip) {
  extern __shared__ float4 tri_smem[];
  TriSmem& sm = *reinterpret_cast<TriSmem*>(tri_smem);
  __shared__ int s_tk;
  if (skip && *skip) return;
  const int G = int(ceil_div(R, kCG)), nblk = int(ceil_div(n, kB));
  __shared__ uint8_t s_after[kMaxBlocks];
  if (threadIdx.x == 0) s_tk = atomicAdd(ticket, 1);
  for (int i = threadIdx.x; i < nblk; i += kTriThreads) s_after[i] = uint8_t(after[i]);  // beside the ticket's latency
  __syncthreads();
  const int t = s_tk / G, cbase = (s_tk % G) * kCG;
  if (t >= nblk) return;
  if (s_after[LOWER ? t : nblk - 1 - t])
    tri_block<LOWER, true>(sm, t, cbase, Gh, Gl, ldg, tiles, n, R, Bin, perm, win, wout, Y, accumulate, st);
  else
    tri_block<LOWER, false>(sm, t, cbase, Gh, Gl, ldg, tiles, n, R, Bin, perm, win, wout, Y, accumulate, st);
}

// ---------------------------------------------------------------------------
struct BatchWs {
  BatchHeader* hdr;
  float *Gh, *Gl, *tilesL, *tilesU;  // premultiplied factors, inverted diagonal blocks
  double *invL, *invU, *Bs, *X, *D, *partial, *chunk, *KP, *VP;
  int32_t *afterL, *afterU;  // which block rows take the second form
  Word* words;  // tickets (the first word), then the words of both solves
  void *Kd, *Vd, *columns;  // digits of Ks, of the value matrix, of a multiplied block
};

size_t batch_layout(int n, char* base, BatchWs* w) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = (off + 255) & ~size_t(255);
    char* p = base ? base + off : nullptr;
    off += bytes;
    return p;
  };
  const int64_t ld = updes_matrix_ld(n, 8);
  const size_t v = size_t(n) * kMaxR * sizeof(double), nblk = size_t(ceil_div(n, kB));
  BatchWs b;
  b.hdr = reinterpret_cast<BatchHeader*>(take(sizeof(BatchHeader)));
  b.Gh = reinterpret_cast<float*>(take(size_t(n) * ld * sizeof(float)));
  b.Gl = reinterpret_cast<float*>(take(size_t(n) * ld * sizeof(float)));
  b.tilesL = reinterpret_cast<float*>(take(nblk * kTilePlanes * kB * kB * sizeof(float)));
  b.tilesU = reinterpret_cast<float*>(take(nblk * kTilePlanes * kB * kB * sizeof(float)));
  b.afterL = reinterpret_cast<int32_t*>(take(nblk * sizeof(int32_t)));
  b.afterU = reinterpret_cast<int32_t*>(take(nblk * sizeof(int32_t)));
  b.invL = reinterpret_cast<double*>(take(nblk * kB * kB * sizeof(double)));
  b.invU = reinterpret_cast<double*>(take(nblk * kB * kB * sizeof(double)));
  b.Bs = reinterpret_cast<double*>(take(v));
  b.X = reinterpret_cast<double*>(take(v));
  b.D = reinterpret_cast<double*>(take(v));
  b.words = reinterpret_cast<Word*>(take((1 + 2 * size_t(n) * kMaxR) * sizeof(Word)));
  b.partial = reinterpret_cast<double*>(take(kRhs64MaxSplits * v));
  b.chunk = reinterpret_cast<double*>(take(size_t(kChunk) * ld * sizeof(double)));
  b.KP = reinterpret_cast<double*>(take(size_t(n) * kMaxM * sizeof(double)));
  b.VP = reinterpret_cast<double*>(take(size_t(n) * kMaxM * sizeof(double)));
  b.Kd = take(rhs64_matrix_bytes(n, n));
  b.Vd = take(rhs64_matrix_bytes(n, n));
  b.columns = take(rhs64_columns_bytes(n));
  if (w) *w = b;
  return off + 256;
}

// Opt the kernels into their dynamic shared memory on the current device (once per device; host calls that are not
// stream operations, made before the first launch).
int batch_kernel_setup() {
  static std::atomic<unsigned long long> done[8];
  const void* tri[] = {(const void*)batch_tri_kernel<true>, (const void*)batch_tri_kernel<false>};
  const void* inv[] = {(const void*)tri_inverse_kernel<double, true>, (const void*)tri_inverse_kernel<double, false>,
                       (const void*)tri_inverse_kernel<float, true>,  (const void*)tri_inverse_kernel<float, false>,
                       (const void*)tri_premultiply_kernel<double>,   (const void*)tri_premultiply_kernel<float>};
  for (int i = 0; i < 2; ++i)
    if (int e = smem_opt_in(tri[i], int(sizeof(TriSmem)), done[i])) return e;
  for (int i = 0; i < 6; ++i)
    if (int e = smem_opt_in(inv[i], int(sizeof(InverseSmem)), done[2 + i])) return e;
  return rhs64_setup();
}

}  // namespace

int value_rows(const updes_problem* p, int r0, int rows, double* out, int64_t ld, cudaStream_t s);

// Views of the solve workspace the batch needs (defined in solve.cu).
int solve_ws_views(const updes_problem* p, void* workspace, size_t workspace_bytes, const float** Khi,
                   const float** Klo, const float** F32, const double** F64, int64_t* ld, const int32_t** piv,
                   const double** dr, const double** dc, DeviceStatus** st, const int32_t** state);

namespace {

// The inverted diagonal blocks and the premultiplied block rows of the factors F.
template <typename TF>
int prepare_factors(int n, const TF* F, int64_t ld, const BatchWs& b, cudaStream_t s) {
  const unsigned nblk = unsigned(ceil_div(n, kB));
  tri_inverse_kernel<TF, true><<<nblk, 256, sizeof(InverseSmem), s>>>(F, ld, n, b.invL, b.tilesL, b.afterL);
  UPDES_LAUNCH_CHECK();
  tri_inverse_kernel<TF, false><<<nblk, 256, sizeof(InverseSmem), s>>>(F, ld, n, b.invU, b.tilesU, b.afterU);
  UPDES_LAUNCH_CHECK();
  tri_premultiply_kernel<TF><<<dim3(nblk, nblk), 256, sizeof(InverseSmem), s>>>(F, ld, n, b.invL, b.invU, b.afterL,
                                                                                 b.afterU, b.Gh, b.Gl);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

// Y (+)= M^-1 B for n x R blocks (permute, L, U).
int batch_precond(int n, int R, const BatchWs& b, int64_t ld, const int32_t* piv, const double* B, double* Y,
                  bool accumulate, DeviceStatus* st, cudaStream_t s, const int32_t* skip = nullptr) {
  const unsigned grid = unsigned(ceil_div(n, kB) * ceil_div(R, kCG));
  StatScope sc(kStatTrsv, s, 2.0 * n * n * R, double(n) * n * 8.0);
  int* tickets = reinterpret_cast<int*>(b.words);
  Word *wL = b.words + 1, *wU = wL + size_t(n) * R;
  UPDES_CUDA_TRY(cudaMemsetAsync(b.words, 0, (1 + 2 * size_t(n) * R) * sizeof(Word), s));
  batch_tri_kernel<true><<<grid, kTriThreads, sizeof(TriSmem), s>>>(b.Gh, b.Gl, ld, b.tilesL, b.afterL, n, R, B, piv + n, nullptr, wL,
                                                            nullptr, 0, tickets, st, skip);
  UPDES_LAUNCH_CHECK();
  batch_tri_kernel<false><<<grid, kTriThreads, sizeof(TriSmem), s>>>(b.Gh, b.Gl, ld, b.tilesU, b.afterU, n, R, nullptr, nullptr, wL, wU, Y,
                                                             accumulate, tickets + 1, st, skip);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

}  // namespace

extern "C" int updes_batch_workspace(int32_t n, size_t* bytes) {
  if (n <= 0 || !bytes) return UPDES_ERR_INVALID;
  *bytes = batch_layout(n, nullptr, nullptr);
  return UPDES_OK;
}

extern "C" int updes_batch_prepare(const updes_problem* p, void* workspace, size_t workspace_bytes, void* batch_ws,
                                   size_t batch_ws_bytes, void* stream) {
  if (!p || !batch_ws) return UPDES_ERR_INVALID;
  const int n = p->N + p->M;
  if (ceil_div(n, kB) > kMaxBlocks) return UPDES_ERR_UNSUPPORTED;
  if (batch_ws_bytes < batch_layout(n, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  const float *Khi, *Klo, *F32;
  const double *F64, *dr, *dc;
  const int32_t *piv, *state;
  int64_t ld;
  DeviceStatus* st;
  int e = solve_ws_views(p, workspace, workspace_bytes, &Khi, &Klo, &F32, &F64, &ld, &piv, &dr, &dc, &st, &state);
  if (e) return e;
  if ((e = batch_kernel_setup())) return e;
  BatchWs b;
  batch_layout(n, static_cast<char*>(batch_ws), &b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int32_t h[4];
  UPDES_CUDA_TRY(cudaMemcpyAsync(h, state, sizeof h, cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  if (h[0] != n || h[2] != 1) return UPDES_ERR_INVALID;  // no factorisation of this system in the workspace
  if ((e = h[1] == UPDES_PREC_FP64 ? prepare_factors(n, F64, ld, b, s) : prepare_factors(n, F32, ld, b, s))) return e;
  if ((e = rhs64_matrix(nullptr, Khi, Klo, ld, n, p->N, 0, n, b.Kd, s))) return e;
  polynomial_columns_kernel<<<unsigned(ceil_div(int64_t(n) * p->M, 256)), 256, 0, s>>>(Khi, Klo, ld, p->nodes, n, p->N, b.KP,
                                                                                     b.VP);
  UPDES_LAUNCH_CHECK();
  if (!p->supports)  // values on local supports have no batched form
    for (int r0 = 0; r0 < p->N; r0 += kChunk) {
      const int rows = std::min(kChunk, p->N - r0);
      if ((e = value_rows(p, r0, rows, b.chunk, ld, s))) return e;
      if ((e = rhs64_matrix(b.chunk, nullptr, nullptr, ld, p->N, p->N, r0, rows, b.Vd, s))) return e;
    }
  const BatchHeader hd{n, h[1], 1, h[3], p->N, p->supports ? 0 : 1};
  UPDES_CUDA_TRY(cudaMemcpyAsync(b.hdr, &hd, sizeof hd, cudaMemcpyHostToDevice, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return UPDES_OK;
}

extern "C" int updes_solve_batch(const updes_problem* p, int32_t R, const double* Q, int64_t ldq, double* coeffs,
                                 int64_t ldc, int32_t sweeps, void* workspace, size_t workspace_bytes,
                                 void* batch_ws, size_t batch_ws_bytes, void* stream) {
  if (!p || R <= 0 || R > kMaxR || !Q || !coeffs || ldq < R || ldc < R || sweeps < 0 || !batch_ws)
    return UPDES_ERR_INVALID;
  const int n = p->N + p->M;
  if (ceil_div(n, kB) > kMaxBlocks) return UPDES_ERR_UNSUPPORTED;
  if (batch_ws_bytes < batch_layout(n, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  const float *Khi, *Klo, *F32;
  const double *F64, *dr, *dc;
  const int32_t *piv, *state;
  int64_t ld;
  DeviceStatus* st;
  int e = solve_ws_views(p, workspace, workspace_bytes, &Khi, &Klo, &F32, &F64, &ld, &piv, &dr, &dc, &st, &state);
  if (e) return e;
  if ((e = batch_kernel_setup())) return e;
  BatchWs b;
  batch_layout(n, static_cast<char*>(batch_ws), &b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t total = int64_t(n) * R;
  const unsigned g = unsigned(ceil_div(total, 256));
  batch_rhs_kernel<<<g, 256, 0, s>>>(Q, ldq, p->N, n, R, dr, b.Bs, state, b.hdr, st);
  UPDES_LAUNCH_CHECK();
  if ((e = batch_precond(n, R, b, ld, piv, b.Bs, b.X, false, st, s))) return e;
  const int splits = rhs64_splits(n, p->N);
  // FP64 factors (precision 0 in the header) get a sweep in any case, see kPremultiplied; the kernels read which they are
  static_assert(UPDES_PREC_FP64 == 0, "skip");
  const int32_t* skip = sweeps == 0 ? &b.hdr->precision : nullptr;
  for (int it = 0; it < std::max(sweeps, 1); ++it) {
    {
      StatScope sc(kStatGemv, s, 2.0 * n * n * R, 14.0 * n * double(n));
      if ((e = rhs64_multiply(b.Kd, n, p->N, b.X, R, R, b.columns, b.partial, splits, st, s, skip)))
        return e;
      batch_residual_kernel<<<g, 256, 0, s>>>(b.Bs, b.partial, splits, n, p->N, R, b.KP, b.X, b.D, skip);
      UPDES_LAUNCH_CHECK();
    }
    if ((e = batch_precond(n, R, b, ld, piv, b.D, b.X, true, st, s, skip))) return e;
  }
  batch_unscale_kernel<<<g, 256, 0, s>>>(b.X, dc, n, R, coeffs, ldc);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

extern "C" int updes_eval_values_prepared(const updes_problem* p, int32_t R, const double* C, int64_t ldc, double* vals,
                                          int64_t ldv, void* workspace, size_t workspace_bytes, void* batch_ws,
                                          size_t batch_ws_bytes, void* stream) {
  if (!p || !C || !vals || R <= 0 || R > kMaxR || ldc < R || ldv < R || !batch_ws) return UPDES_ERR_INVALID;
  if (p->supports) return UPDES_ERR_UNSUPPORTED;
  const int n = p->N + p->M;
  if (batch_ws_bytes < batch_layout(n, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  const float *Khi, *Klo, *F32;
  const double *F64, *dr, *dc;
  const int32_t *piv, *state;
  int64_t ld;
  DeviceStatus* st;
  int e = solve_ws_views(p, workspace, workspace_bytes, &Khi, &Klo, &F32, &F64, &ld, &piv, &dr, &dc, &st, &state);
  if (e) return e;
  BatchWs b;
  batch_layout(n, static_cast<char*>(batch_ws), &b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int splits = rhs64_splits(p->N, p->N);
  if ((e = rhs64_multiply(b.Vd, p->N, p->N, C, ldc, R, b.columns, b.partial, splits, st, s))) return e;
  batch_values_kernel<<<unsigned(ceil_div(int64_t(p->N) * R, 256)), 256, 0, s>>>(
      b.partial, splits, p->N, n, R, b.VP, C, ldc, vals, ldv, state, b.hdr, st);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}
