// Public LU / solve entry points and the GMRES-refined collocation solve.
//
// updes_solve replaces pde_solver's assemble_B -> lineax QR ->
// core_compute_coefficients sequence (updes/operators.py:602-618) by one
// factorisation of the augmented Kansa matrix K and refinement in FP64.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "common.cuh"
#include "gemm_tc.cuh"
#include "lu.cuh"
#include "stats.cuh"

int updes_check_problem(const updes_problem* p);
size_t eval_values_sym_bytes(int N);
int eval_values_sym(const updes_problem* p, const double* coeffs, double* vals, double* part, cudaStream_t s,
                    bool df);

namespace {

std::mutex g_err_mu;
std::string g_last_error;

constexpr int kMaxPermN = 51200;  // interchanges read from shared memory

// perm[i] = the row that the interchanges k <-> piv[k] >= k, k = 0 .. n-1, bring to position i: a thread follows its
// position backwards through them.  Those after step i do not touch it, step i takes it to piv[i], and each earlier one
// that ends where it stands takes it to k.  A chain of one comparison per step, four steps a shared-memory read, for all positions side
// by side; applied one after the other by one thread the interchanges took 33 ns each (0.33 ms at n = 10,006).
__global__ void __launch_bounds__(128) perm_from_piv_kernel(const int32_t* __restrict__ piv, int n,
                                                            int32_t* __restrict__ perm) {
  extern __shared__ __align__(16) int32_t sp[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x, top = min(n, int((blockIdx.x + 1) * blockDim.x));
  for (int k = threadIdx.x; k < top; k += blockDim.x) sp[k] = piv[k];
  __syncthreads();
  if (i >= n) return;
  int r = sp[i];
  int k = i - 1;
  for (; (k & 3) != 3 && k >= 0; --k)
    if (r == sp[k]) r = k;
  for (; k >= 0; k -= 4) {
    const int4 p = *reinterpret_cast<const int4*>(sp + k - 3);
    if (r == p.w) r = k;
    if (r == p.z) r = k - 1;
    if (r == p.y) r = k - 2;
    if (r == p.x) r = k - 3;
  }
  perm[i] = r;
}

// out[i] = scale[i] * in[perm[i]] (gather, scale may be null) or out[perm[i]] = in[i] (scatter)
__global__ void permute_kernel(double* __restrict__ out, const double* __restrict__ in, int64_t in_stride,
                               int64_t out_stride, const int32_t* __restrict__ perm, int n, int scatter) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (scatter) out[int64_t(perm[i]) * out_stride] = in[int64_t(i) * in_stride];
  else out[int64_t(i) * out_stride] = in[int64_t(perm[i]) * in_stride];
}

// A power of two that brings the maximum m into [1/2, 1) (scaling by it is exact); 1 for m = 0 or a non-finite m.
__device__ __forceinline__ double pow2_scale(double m) {
  int e = 0;
  if (m > 0.0 && isfinite(m)) frexp(m, &e);
  return ldexp(1.0, -e);
}

// Scaling of the FP64 factorisation.  Its digit products (gemm_tc64.cu) share one power of two along a row of L and a column
// of U, so the entries that meet there have to be of one size.  In K = [[op Phi, op P], [P^T, 0]] of a domain of side S they
// are not: Phi is S^(2a+1) beside the ones of P, and scaled by the whole row's and column's largest entry, the ones, it
// stays so.  So the kernel block's rows and columns are scaled to their own maxima, the polynomial ones to the
// size that the constant then has beside these (polynomial_scale_kernel), and only then whole rows and columns: whatever the
// side, a matrix like the unit square's.  r^3, 600 nodes, side 2^-10: nodal values wrong by 1.6e-7 with whole rows
// and columns alone, by 4e-14 (as on the unit square) with this.

// Only exponents count, so the passes over K compare those, on integers: the FP64 pipe takes 64 cycles an operation and warp
// and made a pass 0.6 ms at n = 10,006, memory 0.15.

// e with |v| in [2^(e-1), 2^e); kNoExp for 0 and subnormal numbers.
constexpr int kNoExp = -(1 << 20);
__device__ __forceinline__ int exponent_of(double v) {
  const int f = (__double2hiint(v) >> 20) & 0x7ff;
  return f ? f - 1022 : kNoExp;
}
// the power of two that brings a maximum with that exponent into [1/2, 1); 1 for 0 and for infinities
__device__ __forceinline__ double scale_by(int e) { return e <= kNoExp / 2 || e >= 1025 ? 1.0 : ldexp(1.0, -e); }

// dr[i], i < rows, by the largest of the first `cols` entries, or, where these lie below 2^-400 of the largest of all n, by
// that; entries of column j times dc[j] (dc may be null).
__global__ void __launch_bounds__(256) row_scale_kernel(const double* __restrict__ K, int64_t ld, int n, int rows, int cols,
                                                        const double* __restrict__ dc, double* __restrict__ dr) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= rows) return;
  const double2* row = reinterpret_cast<const double2*>(K + int64_t(i) * ld);
  int m = kNoExp, all = kNoExp;
  for (int j0 = 2 * lane; j0 < n; j0 += 256) {  // four loads of two entries in flight
    double2 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = j0 + 64 * u < n ? row[j0 / 2 + 32 * u] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + 64 * u + h;
        if (j >= n) continue;
        const int e = exponent_of(h ? v[u].y : v[u].x) + (dc ? exponent_of(dc[j]) - 1 : 0);
        if (j < cols) m = max(m, e);
        all = max(all, e);
      }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  all = __reduce_max_sync(0xffffffffu, all);
  if (lane == 0) dr[i] = scale_by(m > all - 400 ? m : all);
}

// The polynomial columns (blockIdx.x == 0) or rows of K, all by one power of two: the constant's entries in the first N rows
// (columns), with the scales of these, brought to a geometric mean of 1 where that is above, beside kernel entries of up to 1.
// One factor for all, because monomials that are large among themselves (nodes far from the origin) are better left so:
// 36 x 24 nodes around 100, Gaussian, 1.3e-11 with each at 1, 5.8e-13 with whole rows.  Not by the largest entry: a
// few nodes far from the others have kernel rows of 1e-10 and, scaled to 1, a constant of 1e10; made 1, it leaves all
// other nodes' at 1e-10 and the polynomial wrong by 1.6e-6 (20 x 16 nodes, one facet far away; with the mean, 2.6e-12).
__global__ void __launch_bounds__(256) polynomial_scale_kernel(const double* __restrict__ K, int64_t ld, int N, int M,
                                                               double* __restrict__ dr, double* __restrict__ dc) {
  __shared__ int sum_s, count_s;
  const bool columns = blockIdx.x == 0;
  if (threadIdx.x == 0) sum_s = count_s = 0;
  __syncthreads();
  int sum = 0, count = 0;  // of exponents: below 2,200 each
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const int e = exponent_of(columns ? K[int64_t(i) * ld + N] : K[int64_t(N) * ld + i]);
    if (e == kNoExp || e >= 1025) continue;
    sum += e + exponent_of(columns ? dr[i] : dc[i]) - 1;
    ++count;
  }
  atomicAdd(&sum_s, sum);
  atomicAdd(&count_s, count);
  __syncthreads();
  const int e = count_s ? max(__double2int_rn(double(sum_s) / count_s), 0) : 0;
  if (threadIdx.x < M) (columns ? dc : dr)[N + threadIdx.x] = ldexp(1.0, -e);
}

// Largest exponents of the columns of |K| diag(dr) over a chunk of the first `rows` rows per blockIdx.y, plus kExpBias, into
// the low words of colmax, which must start at zero; column_scale_kernel then makes dc of them in place.
constexpr int kColScaleChunks = 64;
constexpr int kExpBias = 8192;
__global__ void __launch_bounds__(256) column_exponents_kernel(const double* __restrict__ K, int64_t ld, int n, int rows,
                                                               const double* __restrict__ dr, int2* __restrict__ colmax) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int chunk = int(ceil_div(rows, kColScaleChunks));
  const int i0 = blockIdx.y * chunk, i1 = min(rows, i0 + chunk);
  int m = kNoExp;
  for (int i = i0; i < i1; i += 8) {  // eight loads in flight
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = i + u < i1 ? K[int64_t(i + u) * ld + j] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i + u < i1) m = max(m, exponent_of(v[u]) + exponent_of(dr[i + u]) - 1);
  }
  if (m > kNoExp / 2) atomicMax(&colmax[j].x, m + kExpBias);
}
__global__ void column_scale_kernel(int n, double* __restrict__ dc) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int m = reinterpret_cast<const int2*>(dc)[j].x;
  dc[j] = m ? scale_by(m - kExpBias) : 1.0;
}

// dc_j = 2^-e with max_i |K_ij| dr_i in [2^(e-1), 2^e)  (dc holds the maxima' bits on entry)
__global__ void col_scale_kernel(int n, double* __restrict__ dc) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double m = __longlong_as_double((long long)reinterpret_cast<unsigned long long*>(dc)[j]);
  dc[j] = pow2_scale(m);
}

// dr[i] = 2^-e with the row maximum (FP32 bit pattern in maxbits) in [2^(e-1), 2^e)
__global__ void row_scale_bits_kernel(const unsigned* __restrict__ maxbits, int n, double* __restrict__ dr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dr[i] = pow2_scale(double(__uint_as_float(maxbits[i])));
}

// Column maxima of |Khi| diag(dr) (the FP32 plane of an unscaled double-float K) over a chunk of rows per
// blockIdx.y, combined with an integer atomicMax on the bit patterns (non-negative doubles order like their bits); colmax
// must start at zero.
__global__ void col_max_f32_kernel(const float* __restrict__ Khi, int64_t ld, int n, const double* __restrict__ dr,
                                   unsigned long long* __restrict__ colmax) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int rows = int(ceil_div(n, kColScaleChunks));
  const int i0 = blockIdx.y * rows, i1 = min(n, i0 + rows);
  // eight independent loads in flight per thread (the column walk is otherwise one dependent load per row);
  // |hi| dr_i is formed in FP32 (dr is a power of two, exact) and widened once at the end
  float m8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int i = i0;
  for (; i + 8 <= i1; i += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = __ldg(Khi + int64_t(i + u) * ld + j);
#pragma unroll
    for (int u = 0; u < 8; ++u) m8[u] = fmaxf(m8[u], fabsf(v[u]) * float(dr[i + u]));
  }
  for (; i < i1; ++i) m8[0] = fmaxf(m8[0], fabsf(__ldg(Khi + int64_t(i) * ld + j)) * float(dr[i]));
  float mf = m8[0];
#pragma unroll
  for (int u = 1; u < 8; ++u) mf = fmaxf(mf, m8[u]);
  const double m = double(mf);
  if (m > 0.0) atomicMax(colmax + j, (unsigned long long)__double_as_longlong(m));
}

// Both planes times dr_i dc_j in place (powers of two: exact), four columns a thread, rows strided over grid.y;
// with hi2/lo2 the scaled planes are also written there (the factorisation's working copy, in the same pass).
__global__ void __launch_bounds__(256) scale_planes_kernel(float* __restrict__ hi, float* __restrict__ lo, int64_t ld,
                                                           int n, const double* __restrict__ dr,
                                                           const double* __restrict__ dc, float* __restrict__ hi2,
                                                           float* __restrict__ lo2) {
  const int64_t j0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (j0 >= n) return;
  float cs[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) cs[u] = j0 + u < n ? float(dc[j0 + u]) : 1.f;
  for (int i = blockIdx.y; i < n; i += gridDim.y) {
    const float rs = float(dr[i]);
    float4* ph = reinterpret_cast<float4*>(hi + int64_t(i) * ld + j0);
    float4* pl = reinterpret_cast<float4*>(lo + int64_t(i) * ld + j0);
    float4 h = *ph, l = *pl;
    h.x = h.x * rs * cs[0]; h.y = h.y * rs * cs[1]; h.z = h.z * rs * cs[2]; h.w = h.w * rs * cs[3];
    l.x = l.x * rs * cs[0]; l.y = l.y * rs * cs[1]; l.z = l.z * rs * cs[2]; l.w = l.w * rs * cs[3];
    *ph = h;
    *pl = l;
    if (hi2) {
      *reinterpret_cast<float4*>(hi2 + int64_t(i) * ld + j0) = h;
      *reinterpret_cast<float4*>(lo2 + int64_t(i) * ld + j0) = l;
    }
  }
}

// out_i = dr_i * (bsign * b_i + ksign * sum_j K_ij dc_j x_j), one warp per row (dr, dc, b may be null)
// With absout != null also writes absout_i = dr_i * (sum_j |K_ij dc_j x_j| + |b_i|) (backward-error denominators).
__global__ void __launch_bounds__(256) gemv_kernel(const double* __restrict__ K, int64_t ld, int n,
                                                   const double* __restrict__ x, const double* __restrict__ b,
                                                   const double* __restrict__ dr, const double* __restrict__ dc,
                                                   double bsign, double ksign, double* __restrict__ out,
                                                   double* __restrict__ absout = nullptr) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  const double* row = K + int64_t(warp) * ld;
  double s = 0.0, a = 0.0;
  for (int j = lane; j < n; j += 32) {
    const double t = row[j] * (dc ? dc[j] * x[j] : x[j]);
    s += t;
    a += fabs(t);
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    a += __shfl_xor_sync(0xffffffffu, a, o);
  }
  if (lane == 0) {
    double v = ksign * s + (b ? bsign * b[warp] : 0.0);
    out[warp] = dr ? dr[warp] * v : v;
    if (absout) absout[warp] = (dr ? dr[warp] : 1.0) * (a + (b ? fabs(b[warp]) : 0.0));
  }
}

// Transposed: out_j = dc_j * (bsign * b_j + ksign * sum_i K_ij dr_i x_i), 256 columns per CTA.
__global__ void __launch_bounds__(256) gemv_t_kernel(const double* __restrict__ K, int64_t ld, int n,
                                                     const double* __restrict__ x, const double* __restrict__ b,
                                                     const double* __restrict__ dr, const double* __restrict__ dc,
                                                     double bsign, double ksign, double* __restrict__ out,
                                                     double* __restrict__ absout = nullptr) {
  __shared__ double part[8][33], apart[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  double s = 0.0, a = 0.0;
  if (j < n)
    for (int i = w; i < n; i += 8) {
      const double t = K[int64_t(i) * ld + j] * (dr ? dr[i] * x[i] : x[i]);
      s += t;
      a += fabs(t);
    }
  part[w][lane] = s;
  apart[w][lane] = a;
  __syncthreads();
  if (w == 0 && j < n) {
    double t = 0.0, ta = 0.0;
    for (int q = 0; q < 8; ++q) {
      t += part[q][lane];
      ta += apart[q][lane];
    }
    double v = ksign * t + (b ? bsign * b[j] : 0.0);
    out[j] = dc ? dc[j] * v : v;
    if (absout) absout[j] = (dc ? dc[j] : 1.0) * (ta + (b ? fabs(b[j]) : 0.0));
  }
}

// Double-float matrix-vector products with the equilibrated K stored as FP32 planes (hi, lo):
// exact FP32 products (FMA), compensated sums; the absolute sums for the backward error in FP32.
__device__ __forceinline__ void df_acc(float kh, float kl, float a, float b, float& sh, float& sl, float& sa) {
  const float p = __fmul_rn(kh, a);
  const float e = __fmaf_rn(kh, a, -p);
  const float s = __fadd_rn(sh, p);
  const float bb = __fsub_rn(s, sh);
  float t = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  t = __fadd_rn(t, __fadd_rn(sl, __fmaf_rn(kh, b, __fmaf_rn(kl, a, e))));
  sh = __fadd_rn(s, t);  // renormalise, so the low word never carries more than half an ulp of sh
  sl = __fsub_rn(t, __fsub_rn(sh, s));
  sa = __fadd_rn(sa, fabsf(p));
}

// out_i = ksign * sum_j K_ij x_j (x as FP32 planes xh, xl padded with zeros to ld); absout_i = sum |K_ij x_j|
__global__ void __launch_bounds__(256) gemv_df_kernel(const float* __restrict__ Khi, const float* __restrict__ Klo,
                                                      int64_t ld, int n, const float* __restrict__ xh,
                                                      const float* __restrict__ xl, double ksign,
                                                      double* __restrict__ out, double* __restrict__ absout) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= n) return;
  const float4* kh4 = reinterpret_cast<const float4*>(Khi + int64_t(row) * ld);
  const float4* kl4 = reinterpret_cast<const float4*>(Klo + int64_t(row) * ld);
  const float4* a4 = reinterpret_cast<const float4*>(xh);
  const float4* b4 = reinterpret_cast<const float4*>(xl);
  float sh = 0.f, sl = 0.f, sa = 0.f;
  for (int64_t q = lane; q < ld / 4; q += 32) {
    const float4 kh = kh4[q], kl = kl4[q], a = a4[q], b = b4[q];
    df_acc(kh.x, kl.x, a.x, b.x, sh, sl, sa);
    df_acc(kh.y, kl.y, a.y, b.y, sh, sl, sa);
    df_acc(kh.z, kl.z, a.z, b.z, sh, sl, sa);
    df_acc(kh.w, kl.w, a.w, b.w, sh, sl, sa);
  }
  double v = double(sh) + double(sl);
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(0xffffffffu, v, o);
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
  }
  if (lane == 0) {
    out[row] = ksign * v;
    if (absout) absout[row] = double(sa);
  }
}

// out_j = ksign * sum_i K_ij x_i (transposed), 32 columns per CTA, 8 warps over the rows
__global__ void __launch_bounds__(256) gemv_t_df_kernel(const float* __restrict__ Khi, const float* __restrict__ Klo,
                                                        int64_t ld, int n, const float* __restrict__ xh,
                                                        const float* __restrict__ xl, double ksign,
                                                        double* __restrict__ out, double* __restrict__ absout) {
  __shared__ double part[8][33];
  __shared__ float apart[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  float sh = 0.f, sl = 0.f, sa = 0.f;
  if (j < n)
    for (int i = w; i < n; i += 8) {
      const int64_t idx = int64_t(i) * ld + j;
      df_acc(Khi[idx], Klo[idx], xh[i], xl[i], sh, sl, sa);
    }
  part[w][lane] = double(sh) + double(sl);
  apart[w][lane] = sa;
  __syncthreads();
  if (w == 0 && j < n) {
    double t = 0.0;
    float ta = 0.f;
    for (int q = 0; q < 8; ++q) {
      t += part[q][lane];
      ta += apart[q][lane];
    }
    out[j] = ksign * t;
    if (absout) absout[j] = double(ta);
  }
}

// (xh, xl) = FP32 planes of x (n values, zero padded to ld)
__global__ void split_vec_kernel(const double* __restrict__ x, int n, int64_t ld, float* __restrict__ xh,
                                 float* __restrict__ xl) {
  const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= ld) return;
  const double v = j < n ? x[j] : 0.0;
  const float h = float(v);
  xh[j] = h;
  xl[j] = float(v - double(h));
}

// W = double(hi) + double(lo): the FP64 working matrix from the double-float planes
__global__ void join_df_kernel(const float* __restrict__ hi, const float* __restrict__ lo, double* __restrict__ W,
                               int64_t total) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e < total) W[e] = double(hi[e]) + double(lo[e]);
}

constexpr int kDotBlocks = 120;
// Refinement stops at a componentwise backward error of 256 FP64 unit roundoffs: the residual is formed
// from the double-float planes of K (48 significant bits per entry), which by themselves put the
// measured backward error of an FP64 LU solution at roughly 50-100 unit roundoffs.
constexpr double kBwdFloor = 256.0 * 1.1102230246251565e-16;
// A restart cycle stops its inner iteration once the estimated residual has fallen by this factor, or earlier
// at the requested tolerance or at the reduction that brings the backward error to its floor (at N = 22,500
// the floor comes first and one cycle of 10 iterations converges; 1e-10 and 1e-14 here measured the same).
constexpr double kInnerReduction = 1e-6;

// The last of a grid's CTAs to arrive here (every thread of the CTA gets the answer): it sees what the others wrote
// before.  *cnt is 0 again afterwards.
__device__ __forceinline__ bool last_cta(unsigned* cnt) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(cnt, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// One Gram-Schmidt pass and the sums that the next one needs: w -= V h_in (h_in null: w as it is), then out_i = V_i . w for
// nv vectors or, with `norm`, out_0 = w . w, in one launch: a CTA per chunk of w, the last of them adds the chunks' sums.
// At n = 600 an iteration is mostly such launches (as a product, a sum of its parts and an update each, with the host
// reading three sums, 8 launches and 3 waits; now 3 and 1).
__global__ void __launch_bounds__(256) gram_schmidt_kernel(const double* __restrict__ V, int64_t ldv, int nv,
                                                           const double* __restrict__ h_in, double* w, int n, bool norm,
                                                           double* partial, unsigned* cnt, double* out) {
  __shared__ double red[8];
  const int chunk = int(ceil_div(n, gridDim.x));
  const int lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  if (h_in)
    for (int t = lo + threadIdx.x; t < hi; t += blockDim.x) {
      double s = 0.0;
      for (int i = 0; i < nv; ++i) s = fma(h_in[i], V[int64_t(i) * ldv + t], s);
      w[t] -= s;
    }
  const int nd = norm ? 1 : nv;
  for (int i = 0; i < nd; ++i) {
    double s = 0.0;
    for (int t = lo + threadIdx.x; t < hi; t += blockDim.x) s = fma(norm ? w[t] : V[int64_t(i) * ldv + t], w[t], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int q = 0; q < 8; ++q) t += red[q];
      partial[blockIdx.x * nd + i] = t;
    }
    __syncthreads();
  }
  if (!last_cta(cnt)) return;
  for (int i = threadIdx.x >> 5; i < nd; i += 8) {
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < gridDim.x; b += 32) s += __ldcg(partial + b * nd + i);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) out[i] = s;
  }
}

// r <- b + r (r holds -K x), and out = {max_i |r_i| / (|K||x| + |b|)_i, r . r, b . b}, the last CTA as above.
__global__ void __launch_bounds__(256) residual_kernel(double* r, const double* __restrict__ b,
                                                       const double* __restrict__ absr, const double* __restrict__ bsabs,
                                                       int n, double* partial, unsigned* cnt, double* out) {
  __shared__ double red[3][8];
  double m = 0.0, rr = 0.0, bb = 0.0;
  auto reduce = [&] {
    for (int o = 16; o > 0; o >>= 1) {
      m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      rr += __shfl_xor_sync(0xffffffffu, rr, o);
      bb += __shfl_xor_sync(0xffffffffu, bb, o);
    }
  };
  const int chunk = int(ceil_div(n, gridDim.x));
  const int lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  for (int t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    const double bv = b[t], v = bv + r[t], a = bsabs[t] + absr[t];
    r[t] = v;
    const double q = a > 0.0 ? fabs(v) / a : (fabs(v) > 0.0 ? INFINITY : 0.0);
    m = fmax(m, q != q ? INFINITY : q);
    rr = fma(v, v, rr);
    bb = fma(bv, bv, bb);
  }
  reduce();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { red[0][wid] = m; red[1][wid] = rr; red[2][wid] = bb; }
  __syncthreads();
  if (threadIdx.x == 0) {
    m = rr = bb = 0.0;
    for (int q = 0; q < 8; ++q) { m = fmax(m, red[0][q]); rr += red[1][q]; bb += red[2][q]; }
    partial[blockIdx.x * 3] = m;
    partial[blockIdx.x * 3 + 1] = rr;
    partial[blockIdx.x * 3 + 2] = bb;
  }
  if (!last_cta(cnt) || wid != 0) return;
  m = rr = bb = 0.0;
  for (int c = lane; c < gridDim.x; c += 32) {
    m = fmax(m, __ldcg(partial + c * 3));
    rr += __ldcg(partial + c * 3 + 1);
    bb += __ldcg(partial + c * 3 + 2);
  }
  reduce();
  if (lane == 0) { out[0] = m; out[1] = rr; out[2] = bb; }
}

// w += sign * sum_i h_i V_i ; if out != null writes there instead of w (out = sign * sum_i h_i V_i)
__global__ void multi_axpy_kernel(const double* __restrict__ V, int64_t ldv, int nv, const double* __restrict__ h,
                                  double sign, double* __restrict__ w, double* __restrict__ out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double s = 0.0;
  for (int i = 0; i < nv; ++i) s = fma(h[i], V[int64_t(i) * ldv + t], s);
  if (out) out[t] = sign * s;
  else w[t] += sign * s;
}

__global__ void axpby_kernel(double* y, double a, const double* x, double b, int n,
                             const double* __restrict__ mul) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double v = a * x[t] + b * y[t];
  y[t] = mul ? v * mul[t] : v;
}

__global__ void rhs_kernel(const double* __restrict__ q, int N, int n, const double* __restrict__ dr,
                           double* __restrict__ bs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  bs[t] = (t < N ? q[t] : 0.0) * dr[t];
}

__global__ void abs_kernel(const double* __restrict__ x, double* __restrict__ y, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) y[t] = fabs(x[t]);
}

struct Carve {
  char* base;
  size_t off = 0;
  template <typename T>
  T* take(size_t count) {
    off = (off + 255) & ~size_t(255);
    T* p = reinterpret_cast<T*>(base ? base + off : nullptr);
    off += count * sizeof(T);
    return p;
  }
};

}  // namespace

void updes_set_last_cuda_error(cudaError_t e, const char* what, const char* file, int line) {
  (void)cudaGetLastError();  // the failure is reported here; later checks on this thread start clean
  std::lock_guard<std::mutex> lk(g_err_mu);
  char buf[512];
  snprintf(buf, sizeof buf, "%s: %s (%s:%d)", cudaGetErrorString(e), what, file, line);
  g_last_error = buf;
}

void updes_set_last_error_text(const std::string& text) {
  std::lock_guard<std::mutex> lk(g_err_mu);
  g_last_error = text;
}

std::string updes_last_error_text() {
  std::lock_guard<std::mutex> lk(g_err_mu);
  return g_last_error;
}

extern "C" const char* updes_last_error(void) {
  std::lock_guard<std::mutex> lk(g_err_mu);
  static thread_local std::string copy;
  copy = g_last_error;
  return copy.c_str();
}

extern "C" int updes_version(void) { return 100; }

extern "C" const char* updes_status_string(int status) {
  switch (status) {
    case UPDES_OK: return "ok";
    case UPDES_ERR_INVALID: return "invalid argument";
    case UPDES_ERR_CUDA: return "CUDA runtime error";
    case UPDES_ERR_SINGULAR: return "singular matrix (zero or non-finite pivot)";
    case UPDES_ERR_NOT_CONVERGED: return "iterative refinement did not converge";
    case UPDES_ERR_TIMEOUT: return "a bounded device-side wait timed out";
    case UPDES_ERR_UNSUPPORTED: return "unsupported by this build";
    case UPDES_ERR_WORKSPACE: return "workspace too small";
    case UPDES_ERR_TOO_LARGE: return "n exceeds UPDES_NOALLOC_MAX_N, the fixed scratch of updes_lu_solve_noalloc";
    default: return "unknown status";
  }
}

extern "C" int64_t updes_matrix_ld(int64_t n, int32_t elem_bytes) {
  (void)elem_bytes;
  return (n + 31) / 32 * 32;
}

// ---------------------------------------------------------------------------
// LU entry points
// ---------------------------------------------------------------------------
namespace {

struct LuWs {
  DeviceStatus* st;
  void* panel;
  size_t panel_bytes;
  int* sync;
  double* tmp;
  float* lo;  // lo plane of the double-float working matrix (FP32 precision, when owned here)
};

// lo_plane: reserve the n x ld FP32 lo plane (updes_lu_factor); updes_solve brings its own.
size_t lu_ws_layout(int n, int precision, char* base, LuWs* out, bool lo_plane = true) {
  Carve c{base};
  LuWs w;
  w.st = c.take<DeviceStatus>(1);
  // a mixed solve may fall back to the FP64 factorisation in the same workspace
  const size_t df = precision == UPDES_PREC_FP32 ? lu_df_workspace_bytes(n) : 0;
  w.panel_bytes = (precision == UPDES_PREC_FP32 && lo_plane) ? df : std::max(df, lu_64_workspace_bytes(n));
  w.panel = c.take<char>(w.panel_bytes);
  w.sync = c.take<int>(ceil_div(n, 64) + 2);
  w.tmp = c.take<double>(n);
  w.lo = (precision == UPDES_PREC_FP32 && lo_plane) ? c.take<float>(size_t(n) * updes_matrix_ld(n, 4)) : nullptr;
  if (out) *out = w;
  return c.off + 256;
}

int read_status(DeviceStatus* st, cudaStream_t s, DeviceStatus* host) {
  UPDES_CUDA_TRY(cudaMemcpyAsync(host, st, sizeof(DeviceStatus), cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return UPDES_OK;
}

// hi = float(v), lo = float(v - hi) with v = dr_i K_ij dc_j (scalings exact; dr, dc may be null)
// hi/lo planes of the scaled K (none when hi is null); with write_back the scaled FP64 entry also replaces
// K's (each thread reads and writes only its own entry, so K may be read and written in place; ldk == ld then).
__global__ void split_df_kernel(double* __restrict__ K, int64_t ldk, float* __restrict__ hi,
                                float* __restrict__ lo, int64_t ld, int n, const double* __restrict__ dr,
                                const double* __restrict__ dc, int write_back) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t i = e / ld, j = e % ld;
  if (i >= n) return;
  double v = 0.0;
  if (j < n) {
    v = K[i * ldk + j];
    if (dr) v *= dr[i];
    if (dc) v *= dc[j];
  }
  if (hi) {
    const float h = float(v);
    hi[i * ld + j] = h;
    lo[i * ld + j] = float(v - double(h));
  }
  if (write_back) K[i * ldk + j] = v;
}

int perm_core(int n, int32_t* piv, cudaStream_t s) {
  if (n > kMaxPermN) return UPDES_ERR_UNSUPPORTED;
  static std::atomic<unsigned long long> attr{0};
  if (int e = smem_opt_in((const void*)perm_from_piv_kernel, int(kMaxPermN * sizeof(int32_t)), attr)) return e;
  perm_from_piv_kernel<<<unsigned(ceil_div(n, 128)), 128, size_t(n + 3) / 4 * 16, s>>>(piv, n, piv + n);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

// Mixed LU of a double-float matrix already split into (hi = F, lo).
int factor_df_core(int n, float* hi, float* lo, int64_t ld, int32_t* piv, const LuWs& w, cudaStream_t s) {
  UPDES_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(DeviceStatus), s));
  int e = lu_factor_df(n, hi, lo, ld, piv, w.panel, w.panel_bytes, w.st, s);
  if (e) return e;
  return perm_core(n, piv, s);
}

// scaled: the rows and columns of A are equilibrated (what the FP64 updates on the tensor cores ask for).
int factor_core(int n, double* A, int64_t lda, int precision, void* F, int64_t ldf, int32_t* piv, const LuWs& w,
                cudaStream_t s, bool scaled) {
  if (precision == UPDES_PREC_FP32) {
    if (!w.lo || !F) return UPDES_ERR_INVALID;
    split_df_kernel<<<unsigned(ceil_div(int64_t(n) * ldf, 256)), 256, 0, s>>>(A, lda, static_cast<float*>(F), w.lo,
                                                                              ldf, n, nullptr, nullptr, 0);
    UPDES_LAUNCH_CHECK();
    return factor_df_core(n, static_cast<float*>(F), w.lo, ldf, piv, w, s);
  }
  UPDES_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(DeviceStatus), s));
  int e;
  {
    double* Fd = F ? static_cast<double*>(F) : A;
    if (Fd != A) {
      UPDES_CUDA_TRY(cudaMemcpy2DAsync(Fd, ldf * 8, A, lda * 8, size_t(n) * 8, n, cudaMemcpyDeviceToDevice, s));
      A = Fd;
      lda = ldf;
    }
    e = lu_factor_64(n, A, lda, piv, w.panel, w.panel_bytes, w.st, s, scaled);
  }
  if (e) return e;
  return perm_core(n, piv, s);
}

// x (contiguous, n) <- A^-1 x or A^-T x using the permutation in piv[n, 2n)
template <typename TF>
int solve_core(int n, const TF* F, int64_t ldf, const int32_t* piv, const double* b, double* x, int trans, const LuWs& w,
               cudaStream_t s, const float* dinv = nullptr, float* xh = nullptr, float* xl = nullptr,
               const float* dinv128 = nullptr, unsigned long long* xtag = nullptr) {
  const int32_t* perm = piv + n;
  const unsigned g = unsigned(ceil_div(n, 256));
  if (!trans) {
    permute_kernel<<<g, 256, 0, s>>>(w.tmp, b, 1, 1, perm, n, 0);
    UPDES_LAUNCH_CHECK();
    int e = trsv_impl<TF>(n, F, ldf, w.tmp, 0, w.sync, w.st, s, dinv, xh, xl, dinv128, xtag);
    if (e) return e;
    e = trsv_impl<TF>(n, F, ldf, w.tmp, 1, w.sync, w.st, s, dinv, xh, xl, dinv128, xtag);
    if (e) return e;
    UPDES_CUDA_TRY(cudaMemcpyAsync(x, w.tmp, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
  } else {
    UPDES_CUDA_TRY(cudaMemcpyAsync(w.tmp, b, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
    int e = trsv_impl<TF>(n, F, ldf, w.tmp, 2, w.sync, w.st, s, dinv, xh, xl, dinv128, xtag);
    if (e) return e;
    e = trsv_impl<TF>(n, F, ldf, w.tmp, 3, w.sync, w.st, s, dinv, xh, xl, dinv128, xtag);
    if (e) return e;
    permute_kernel<<<g, 256, 0, s>>>(x, w.tmp, 1, 1, perm, n, 1);
    UPDES_LAUNCH_CHECK();
  }
  return UPDES_OK;
}

int solve_any(int n, const void* F, int64_t ldf, int precision, const int32_t* piv, double* x, int trans,
              const LuWs& w, cudaStream_t s) {
  if (precision == UPDES_PREC_FP64) return solve_core<double>(n, static_cast<const double*>(F), ldf, piv, x, x, trans, w, s);
  return solve_core<float>(n, static_cast<const float*>(F), ldf, piv, x, x, trans, w, s);
}

}  // namespace

extern "C" int updes_lu_workspace(int32_t n, int32_t precision, size_t* bytes) {
  if (n <= 0 || !bytes || (precision != UPDES_PREC_FP64 && precision != UPDES_PREC_FP32)) return UPDES_ERR_INVALID;
  *bytes = lu_ws_layout(n, precision, nullptr, nullptr);
  return UPDES_OK;
}

extern "C" int updes_lu_factor(int32_t n, double* A, int64_t lda, int32_t precision, void* F, int64_t ldf,
                               int32_t* piv, void* workspace, size_t workspace_bytes, int32_t* info, void* stream) {
  if (n <= 0 || !A || lda < n || !piv || !workspace) return UPDES_ERR_INVALID;
  if (precision != UPDES_PREC_FP64 && precision != UPDES_PREC_FP32) return UPDES_ERR_INVALID;
  if (precision == UPDES_PREC_FP32 && (!F || ldf < n || ldf != updes_matrix_ld(n, 4))) return UPDES_ERR_INVALID;
  if (precision == UPDES_PREC_FP64 && F && ldf < n) return UPDES_ERR_INVALID;
  if (workspace_bytes < lu_ws_layout(n, precision, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  LuWs w;
  lu_ws_layout(n, precision, static_cast<char*>(workspace), &w);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int e = factor_core(n, A, lda, precision, F, ldf, piv, w, s, false);
  if (e) return e;
  DeviceStatus h;
  e = read_status(w.st, s, &h);
  if (e) return e;
  if (info) *info = h.lu_info;
  if (h.error) return h.error;
  return UPDES_OK;
}

extern "C" int updes_lu_solve(int32_t n, const void* F, int64_t ldf, int32_t precision, const int32_t* piv,
                              double* b, int32_t nrhs, int64_t ldb, int32_t trans, void* workspace,
                              size_t workspace_bytes, void* stream) {
  if (n <= 0 || !F || ldf < n || !piv || !b || nrhs <= 0 || ldb < nrhs || !workspace) return UPDES_ERR_INVALID;
  if (precision != UPDES_PREC_FP64 && precision != UPDES_PREC_FP32) return UPDES_ERR_INVALID;
  if (workspace_bytes < lu_ws_layout(n, precision, nullptr, nullptr) + size_t(n) * 8 + 256) return UPDES_ERR_WORKSPACE;
  LuWs w;
  size_t used = lu_ws_layout(n, precision, static_cast<char*>(workspace), &w);
  double* col = reinterpret_cast<double*>(static_cast<char*>(workspace) + ((used + 255) & ~size_t(255)));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  UPDES_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(DeviceStatus), s));
  for (int j = 0; j < nrhs; ++j) {
    double* bj = b + j;
    if (nrhs == 1) {
      int e = solve_any(n, F, ldf, precision, piv, bj, trans, w, s);
      if (e) return e;
      continue;
    }
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(col, 8, bj, ldb * 8, 8, n, cudaMemcpyDeviceToDevice, s));
    int e = solve_any(n, F, ldf, precision, piv, col, trans, w, s);
    if (e) return e;
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(bj, ldb * 8, col, 8, 8, n, cudaMemcpyDeviceToDevice, s));
  }
  DeviceStatus h;
  int e = read_status(w.st, s, &h);
  if (e) return e;
  return h.error;
}

extern "C" int updes_residual(int32_t n, const double* K, int64_t ldk, const double* x, const double* b, double* r,
                              int32_t trans, void* stream) {
  if (n <= 0 || !K || ldk < n || !x || !b || !r) return UPDES_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!trans) gemv_kernel<<<unsigned(ceil_div(int64_t(n) * 32, 256)), 256, 0, s>>>(K, ldk, n, x, b, nullptr, nullptr, 1.0, -1.0, r);
  else gemv_t_kernel<<<unsigned(ceil_div(n, 32)), 256, 0, s>>>(K, ldk, n, x, b, nullptr, nullptr, 1.0, -1.0, r);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

// ---------------------------------------------------------------------------
// The full solve
// ---------------------------------------------------------------------------
namespace {

struct SolveWs {
  LuWs lu;
  double *W, *dr, *dc, *bs, *bsabs, *absr, *x, *r, *z, *wv, *V, *Z, *partial, *h;
  double* evp;  // per-tile partial sums of the symmetric value evaluation
  unsigned* cnt;  // CTAs that have arrived at the end of a reduction (0 between them)
  float *Khi, *Klo;  // equilibrated K as double-float planes (kept for the refinement's residuals)
  float *xh, *xl;    // FP32 planes of the vector a GEMV multiplies
  float* F32;  // hi plane = FP32 factors
  float* Wlo;
  float* dinv;     // inverted 64 x 64 diagonal blocks of the FP32 factors (double-float planes)
  float* dinv128;  // the same for 128 x 128 blocks
  unsigned long long* xtag;  // tagged hand-off words of the 128-row triangular solves (2n)
  int32_t* piv;
  int32_t* state;  // [0] n of the factored system, [1] precision of its factors, [2] 1 when valid, [3] generation,
                   // [4] 1 for FP64 factors made by multiply-adds instead of digit products
  int64_t ld;
};

size_t solve_ws_layout(int n, const updes_solve_opts& o, char* base, SolveWs* out) {
  SolveWs w;
  const int64_t ld = updes_matrix_ld(n, 8);
  Carve c{base};
  const size_t lub = lu_ws_layout(n, o.precision, nullptr, nullptr, false);
  char* lubase = c.take<char>(lub);
  if (base) lu_ws_layout(n, o.precision, lubase, &w.lu, false);
  w.ld = ld;
  w.Khi = c.take<float>(2 * size_t(n) * ld);
  w.Klo = w.Khi + size_t(n) * ld;
  w.xh = c.take<float>(ld);
  w.xl = c.take<float>(ld);
  w.W = c.take<double>(size_t(n) * ld);  // FP64 working matrix, or the hi and lo FP32 planes
  w.F32 = reinterpret_cast<float*>(w.W);
  w.Wlo = w.F32 + size_t(n) * ld;
  w.piv = c.take<int32_t>(2 * size_t(n));
  w.state = c.take<int32_t>(64);
  w.dinv = c.take<float>(diag_inverse_bytes(n) / sizeof(float));
  w.dinv128 = c.take<float>(diag_inverse128_bytes(n) / sizeof(float));
  w.evp = c.take<double>(eval_values_sym_bytes(n) / sizeof(double));
  w.dr = c.take<double>(n);
  w.dc = c.take<double>(n);
  w.bs = c.take<double>(n);
  w.bsabs = c.take<double>(n);
  w.absr = c.take<double>(n);
  w.x = c.take<double>(n);
  w.r = c.take<double>(n);
  w.z = c.take<double>(n);
  w.wv = c.take<double>(n);
  const int m = o.restart > 0 ? o.restart : 1;
  w.V = c.take<double>(size_t(m + 1) * n);
  w.partial = c.take<double>(size_t(kDotBlocks) * (m + 2));
  w.h = c.take<double>(2 * (m + 2));  // two passes' coefficients and a norm, or a residual's three sums
  w.cnt = c.take<unsigned>(64);
  w.xtag = c.take<unsigned long long>(2 * size_t(n));
  w.Z = c.take<double>(size_t(m) * n);  // preconditioned basis vectors M^-1 V_j of a restart cycle
  if (out) *out = w;
  return c.off + 256;
}

updes_solve_opts normalise(const updes_solve_opts* o) {
  updes_solve_opts d;
  d.precision = UPDES_PREC_FP32;
  d.max_iters = 200;
  d.restart = 40;
  d.fallback_fp64 = 1;
  d.tol = 1e-13;
  if (o) {
    d = *o;
    if (d.max_iters <= 0) d.max_iters = 200;
    if (d.restart <= 0) d.restart = 40;
    if (d.restart > 200) d.restart = 200;
    if (!(d.tol > 0)) d.tol = 1e-13;
  }
  return d;
}

// h[0..nv) = V[0..nv)^T w (device), then copied to host
struct Timer {
  cudaEvent_t a, b;
  cudaStream_t s;
  bool ok, marked = false;
  explicit Timer(cudaStream_t st) : s(st) {
    ok = cudaEventCreate(&a) == cudaSuccess && cudaEventCreate(&b) == cudaSuccess;
    if (ok) cudaEventRecord(a, s);
  }
  void mark() {  // the end of what is timed, where stop() comes later
    if (ok) marked = cudaEventRecord(b, s) == cudaSuccess;
  }
  double stop() {
    if (!ok) return 0.0;
    if (!marked) cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    ok = false;
    return ms;
  }
  ~Timer() {
    if (ok) {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  }
};

// Ks z = dr .* (K (dc .* z))
// (trans: Ks^T z = dc .* (K^T (dr .* z)))
int gemv_scaled(const SolveWs& w, int n, const double* z, double ksign, double* out, double* absout,
                cudaStream_t s, bool trans) {
  StatScope sc(kStatGemv, s, 2.0 * n * n, 8.0 * n * double(w.ld));
  split_vec_kernel<<<unsigned(ceil_div(w.ld, 256)), 256, 0, s>>>(z, n, w.ld, w.xh, w.xl);
  UPDES_LAUNCH_CHECK();
  if (trans)
    gemv_t_df_kernel<<<unsigned(ceil_div(n, 32)), 256, 0, s>>>(w.Khi, w.Klo, w.ld, n, w.xh, w.xl, ksign, out, absout);
  else
    gemv_df_kernel<<<unsigned(ceil_div(int64_t(n) * 32, 256)), 256, 0, s>>>(w.Khi, w.Klo, w.ld, n, w.xh, w.xl, ksign,
                                                                              out, absout);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

int apply_K(const SolveWs& w, int n, const double* z, double* out, cudaStream_t s, bool trans = false) {
  return gemv_scaled(w, n, z, 1.0, out, nullptr, s, trans);
}

// out = bs - Ks x; on the host, sums = {the componentwise backward error max_i |out_i| / (|Ks| |x| + |bs|)_i, ||out||^2,
// ||bs||^2}.
int residual_scaled(const SolveWs& w, int n, const double* x, double* out, double* sums, cudaStream_t s,
                    bool trans = false) {
  if (int e = gemv_scaled(w, n, x, -1.0, out, w.absr, s, trans)) return e;
  residual_kernel<<<kDotBlocks, 256, 0, s>>>(out, w.bs, w.absr, w.bsabs, n, w.partial, w.cnt, w.h);
  UPDES_LAUNCH_CHECK();
  UPDES_CUDA_TRY(cudaMemcpyAsync(sums, w.h, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return UPDES_OK;
}

int precond(const SolveWs& w, int n, int precision, const double* b, double* x, cudaStream_t s, bool trans = false) {
  if (precision == UPDES_PREC_FP64) return solve_core<double>(n, w.W, w.ld, w.piv, b, x, trans ? 1 : 0, w.lu, s);
  return solve_core<float>(n, w.F32, w.ld, w.piv, b, x, trans ? 1 : 0, w.lu, s, w.dinv, w.xh, w.xl, w.dinv128,
                           w.xtag);
}

[[maybe_unused]] double host_norm(const std::vector<double>& v) {
  double s = 0;
  for (double a : v) s += a * a;
  return std::sqrt(s);
}

// UPDES_TRACE=1 in the environment prints the refinement history to stderr.
bool trace_on() {
  static const bool on = [] {
    const char* v = std::getenv("UPDES_TRACE");
    return v && v[0] == '1';
  }();
  return on;
}

// Restarted, right-preconditioned GMRES on Ks x = bs starting from w.x, in the flexible form: each cycle keeps
// its preconditioned vectors, so that its update x += M^-1 V y is Z y without another preconditioner solve.
int gmres(const SolveWs& w, int n, int precision, const updes_solve_opts& o, updes_solve_info* info,
          cudaStream_t s, bool trans = false) {
  const int m = o.restart;
  const unsigned g = unsigned(ceil_div(n, 256));
  std::vector<double> H(size_t(m + 1) * m), cs(m), sn(m), gv(m + 1), hcol(m + 2), hh(2 * m + 1);
  int e;
  UPDES_CUDA_TRY(cudaMemsetAsync(w.cnt, 0, sizeof(unsigned), s));
  int total = 0, stalls = 0;
  double last_beta = INFINITY;
  for (;;) {
    double sums[3];
    if ((e = residual_scaled(w, n, w.x, w.r, sums, s, trans))) return e;
    const double bwd = sums[0], beta = std::sqrt(sums[1]), bnorm = std::sqrt(sums[2]);
    info->rel_residual = bnorm > 0 ? beta / bnorm : beta;
    info->backward_error = bwd;
    if (trace_on())
      std::fprintf(stderr, "[updes gmres n=%d prec=%d trans=%d] iters=%d rel_residual=%.3e backward_error=%.3e\n", n,
                   precision, int(trans), total, info->rel_residual, bwd);
    if (!(beta == beta)) return UPDES_ERR_NOT_CONVERGED;
    if (beta <= o.tol * bnorm || bwd <= kBwdFloor) {
      info->converged = 1;
      break;
    }
    if (total >= o.max_iters) break;
    if (beta > 0.5 * last_beta) {
      if (++stalls >= 2) break;  // two restart cycles in a row without halving the residual
    } else {
      stalls = 0;
    }
    last_beta = beta;
    // this cycle stops at whichever comes first: the requested tolerance, the reduction one cycle can
    // deliver, or (with a factor 2 to spare) the reduction that brings the backward error to its floor (the
    // ratio backward error / residual norm changes little between cycles)
    const double target = std::max(o.tol * bnorm, beta * std::max(kInnerReduction, 0.5 * kBwdFloor / bwd));
    // V0 = r / beta
    axpby_kernel<<<g, 256, 0, s>>>(w.V, 1.0 / beta, w.r, 0.0, n, nullptr);
    UPDES_LAUNCH_CHECK();
    std::fill(gv.begin(), gv.end(), 0.0);
    gv[0] = beta;
    int j = 0;
    for (; j < m && total < o.max_iters; ++j, ++total) {
      // z_j = M^-1 v_j is kept (flexible GMRES form): the cycle's update is then Z y, with no further solve
      double* vj = w.V + size_t(j) * n;
      double* zj = w.Z + size_t(j) * n;
      if ((e = precond(w, n, precision, vj, zj, s, trans))) return e;
      if ((e = apply_K(w, n, zj, w.wv, s, trans))) return e;
      // CGS2: the two passes' coefficients and the norm of what is left, read together
      const int nv = j + 1;
      for (int pass = 0; pass < 3; ++pass) {
        gram_schmidt_kernel<<<kDotBlocks, 256, 0, s>>>(w.V, n, nv, pass ? w.h + (pass - 1) * nv : nullptr, w.wv, n,
                                                       pass == 2, w.partial, w.cnt, w.h + pass * nv);
        UPDES_LAUNCH_CHECK();
      }
      UPDES_CUDA_TRY(cudaMemcpyAsync(hh.data(), w.h, (2 * nv + 1) * sizeof(double), cudaMemcpyDeviceToHost, s));
      UPDES_CUDA_TRY(cudaStreamSynchronize(s));
      for (int i = 0; i < nv; ++i) hcol[i] = hh[i] + hh[nv + i];
      const double hn = std::sqrt(hh[2 * nv]);
      hcol[j + 1] = hn;
      if (hn > 0) {
        axpby_kernel<<<g, 256, 0, s>>>(w.V + size_t(j + 1) * n, 1.0 / hn, w.wv, 0.0, n, nullptr);
        UPDES_LAUNCH_CHECK();
      }
      // Givens
      for (int i = 0; i < j; ++i) {
        const double t = cs[i] * hcol[i] + sn[i] * hcol[i + 1];
        hcol[i + 1] = -sn[i] * hcol[i] + cs[i] * hcol[i + 1];
        hcol[i] = t;
      }
      const double d = std::hypot(hcol[j], hcol[j + 1]);
      cs[j] = d > 0 ? hcol[j] / d : 1.0;
      sn[j] = d > 0 ? hcol[j + 1] / d : 0.0;
      hcol[j] = d;
      hcol[j + 1] = 0.0;
      gv[j + 1] = -sn[j] * gv[j];
      gv[j] = cs[j] * gv[j];
      for (int i = 0; i <= j; ++i) H[size_t(i) * m + j] = hcol[i];
      if (trace_on())
        std::fprintf(stderr, "[updes gmres]   j=%d estimate=%.3e h_next=%.3e\n", j, std::fabs(gv[j + 1]) / bnorm, hn);
      if (std::fabs(gv[j + 1]) <= target || hn == 0.0) {
        ++j;
        ++total;
        break;
      }
    }
    // y = R^-1 g
    std::vector<double> y(j);
    for (int i = j - 1; i >= 0; --i) {
      double t = gv[i];
      for (int k = i + 1; k < j; ++k) t -= H[size_t(i) * m + k] * y[k];
      y[i] = H[size_t(i) * m + i] != 0 ? t / H[size_t(i) * m + i] : 0.0;
    }
    if (j > 0) {
      UPDES_CUDA_TRY(cudaMemcpyAsync(w.h, y.data(), j * sizeof(double), cudaMemcpyHostToDevice, s));
      multi_axpy_kernel<<<g, 256, 0, s>>>(w.Z, n, j, w.h, 1.0, nullptr, w.z, n);
      UPDES_LAUNCH_CHECK();
      axpby_kernel<<<g, 256, 0, s>>>(w.x, 1.0, w.z, 1.0, n, nullptr);
      UPDES_LAUNCH_CHECK();
      UPDES_CUDA_TRY(cudaStreamSynchronize(s));
    }
  }
  if (precision == UPDES_PREC_FP32) info->iters = total;
  return UPDES_OK;
}

}  // namespace

extern "C" int updes_solve_workspace(const updes_problem* p, const updes_solve_opts* opts, size_t* bytes) {
  if (updes_check_problem(p) || !bytes) return UPDES_ERR_INVALID;
  const updes_solve_opts o = normalise(opts);
  updes_solve_opts o64 = o;
  o64.precision = UPDES_PREC_FP32;  // the FP64 fallback fits in the same layout
  *bytes = solve_ws_layout(p->N + p->M, o64, nullptr, nullptr);
  return UPDES_OK;
}

namespace {

// out = |T| |v| for one triangle T of the factors in F (row-major), L with its unit diagonal: by rows, a warp each, or
// transposed, a block for 32 columns.  from: v_i is v[from[i]].  With r, also *worst, the largest |r_i| / out_i, r_i being
// r[to[i]] (an order of non-negative doubles is that of their bits).  Bound by the one read of the triangle; it runs only on
// solutions whose backward error is large already.
template <bool TRANS>
__global__ void __launch_bounds__(256) abs_triangle_kernel(const double* __restrict__ F, int64_t ld, int n, bool lower,
                                                           const double* __restrict__ v, const int32_t* __restrict__ from,
                                                           double* __restrict__ out, const double* __restrict__ r,
                                                           const int32_t* __restrict__ to, unsigned long long* worst) {
  __shared__ double part[8][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = TRANS ? blockIdx.x * 32 + lane : blockIdx.x * 8 + wid;  // of out
  auto at = [&](int j) { return fabs(v[from ? from[j] : j]); };
  double sum = 0.0;
  if (i < n) {
    // the entries off the diagonal are before it in L's rows and U's columns, behind it in U's rows and L's columns
    const bool before = lower != TRANS;
    const int j0 = before ? 0 : i + 1, j1 = before ? i : n;
    const int64_t step = TRANS ? ld : 1;
    const double* f = F + (TRANS ? int64_t(i) : int64_t(i) * ld);
    for (int j = j0 + (TRANS ? wid : lane); j < j1; j += TRANS ? 8 : 32) sum = fma(fabs(f[j * step]), at(j), sum);
  }
  if (TRANS) {
    part[wid][lane] = sum;
    __syncthreads();
    if (wid != 0) return;
    for (int q = 1; q < 8; ++q) sum += part[q][lane];
  } else {
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane != 0) return;
  }
  if (i >= n) return;
  sum = fma(lower ? 1.0 : fabs(F[int64_t(i) * ld + i]), at(i), sum);
  out[i] = sum;
  if (r) {
    const double a = fabs(r[to ? to[i] : i]);
    atomicMax(worst, static_cast<unsigned long long>(__double_as_longlong(a != 0.0 ? a / sum : 0.0)));
  }
}

// *worst = max_i |r_i| / (P^T |L| |U| |x|)_i (trans: (|U^T| |L^T| P |x|)_i) for the FP64 factors and the residual r and
// solution x that gmres left: what multiply-adds keep below a small multiple of u, however K is graded.
int residual_by_factors(const SolveWs& w, int n, bool trans, double* worst, cudaStream_t s) {
  const int32_t* perm = w.piv + n;
  unsigned long long* dev = reinterpret_cast<unsigned long long*>(w.h);
  UPDES_CUDA_TRY(cudaMemsetAsync(dev, 0, sizeof *dev, s));
  const unsigned rows = unsigned(ceil_div(n, 8)), columns = unsigned(ceil_div(n, 32));
  if (trans) {
    abs_triangle_kernel<true><<<columns, 256, 0, s>>>(w.W, w.ld, n, true, w.x, perm, w.z, nullptr, nullptr, nullptr);
    UPDES_LAUNCH_CHECK();
    abs_triangle_kernel<true><<<columns, 256, 0, s>>>(w.W, w.ld, n, false, w.z, nullptr, w.wv, w.r, nullptr, dev);
  } else {
    abs_triangle_kernel<false><<<rows, 256, 0, s>>>(w.W, w.ld, n, false, w.x, nullptr, w.z, nullptr, nullptr, nullptr);
    UPDES_LAUNCH_CHECK();
    abs_triangle_kernel<false><<<rows, 256, 0, s>>>(w.W, w.ld, n, true, w.z, nullptr, w.wv, w.r, perm, dev);
  }
  UPDES_LAUNCH_CHECK();
  UPDES_CUDA_TRY(cudaMemcpyAsync(worst, dev, sizeof *worst, cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return UPDES_OK;
}

constexpr int kStateInts = 5;

// When factors from digit products are not trusted: K is then factored again by FP64 multiply-adds, whatever its rows and
// columns look like.  Where the scaled K is still graded (Gaussian kernels that decouple most of the nodes, two clusters of
// very different spacing) the digits can lose what multiply-adds keep: 22 x 16 nodes, one half squeezed to 0.03,
// values wrong by 1e-2 instead of 1.3e-14 (Gaussian), by 2.2e-6 instead of 1.4e-7 (r^5).  The backward error is then above
// 1,024 u, 1.7e-13 and more (the kernels and clouds in use: 2e-15 to 1.1e-13).  But a flat Gaussian, singular to working
// precision, leaves it there too, whatever the factors are made of, so the residual is also compared with what the factors'
// own size lets multiply-adds leave.  In u: 158 flat Gaussians 2 to 25 from digits, 3 to 23 from multiply-adds; graded
// kernels 82 to 1e13 (260 and above where the values suffer) and 15 to 69, of which the 48-bit planes of K and x in the
// residual are up to 64.  512 uneven clouds, half of them flat Gaussians, eight streams: 1.87 s by the backward error alone,
// 1.27 with both, as without any check.
constexpr double kDigitsBackwardError = 0x1p-43;
constexpr double kDigitsResidual = 128 * 0x1p-53;

// Whether the digits' factors have to be made again, after gmres left x and r.
int digits_failed(const SolveWs& w, int n, bool trans, const updes_solve_info& info, bool* failed, cudaStream_t s) {
  *failed = false;
  if (!(info.backward_error > kDigitsBackwardError)) return UPDES_OK;
  double worst = 0.0;
  if (int e = residual_by_factors(w, n, trans, &worst, s)) return e;
  *failed = !(worst <= kDigitsResidual);
  if (trace_on()) std::fprintf(stderr, "[updes solve n=%d] residual of the factors' size: %.1f u\n", n, worst * 0x1p53);
  return UPDES_OK;
}

// Factors of the equilibrated K (double-float planes) at `precision`; records the factored state.
// planes_ready: the working copy already holds the equilibrated K, written by the assembly: for FP32 factors
// the planes F32 and Wlo (double-float assembly), for FP64 factors the FP64 matrix W.
int factor_launch(const SolveWs& w, int n, int precision, cudaStream_t s, bool planes_ready, bool multiply_adds = false) {
  int e;
  UPDES_CUDA_TRY(cudaMemsetAsync(w.state, 0, kStateInts * sizeof(int32_t), s));  // invalid until the factors are complete
  const int64_t total = int64_t(n) * w.ld;
  if (precision == UPDES_PREC_FP64) {
    if (!planes_ready) {
      join_df_kernel<<<unsigned(ceil_div(total, 256)), 256, 0, s>>>(w.Khi, w.Klo, w.W, total);
      UPDES_LAUNCH_CHECK();
    }
    e = factor_core(n, w.W, w.ld, precision, nullptr, w.ld, w.piv, w.lu, s, !multiply_adds);
  } else {
    if (!planes_ready) {
      UPDES_CUDA_TRY(cudaMemcpyAsync(w.F32, w.Khi, size_t(total) * 4, cudaMemcpyDeviceToDevice, s));
      UPDES_CUDA_TRY(cudaMemcpyAsync(w.Wlo, w.Klo, size_t(total) * 4, cudaMemcpyDeviceToDevice, s));
    }
    e = factor_df_core(n, w.F32, w.Wlo, w.ld, w.piv, w.lu, s);
    if (!e) e = diag_inverse(n, w.F32, w.ld, w.dinv, s);
    if (!e) e = diag_inverse128(n, w.F32, w.ld, w.dinv, w.dinv128, s);
  }
  return e;
}

// Waits for what factor_launch issued, reports on it and marks the factors as complete.
int factor_finish(const SolveWs& w, int n, int precision, updes_solve_info* info, cudaStream_t s, Timer& t,
                  bool multiply_adds = false) {
  int e;
  DeviceStatus h;
  if ((e = read_status(w.lu.st, s, &h))) return e;
  if (h.error) return h.error;
  info->lu_info = h.lu_info;
  info->t_factor_ms += t.stop();
  // {n, precision, valid, generation, multiply_adds}: the generation tells derived copies of these factors (the batched
  // solves' double-float planes) that they are stale after a refactorisation
  static std::atomic<int32_t> generation{0};
  const int32_t state[kStateInts] = {n, precision, 1, generation.fetch_add(1) + 1, multiply_adds};
  UPDES_CUDA_TRY(cudaMemcpyAsync(w.state, state, sizeof state, cudaMemcpyHostToDevice, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return UPDES_OK;
}

int factor_stage(const SolveWs& w, int n, int precision, updes_solve_info* info, cudaStream_t s, bool planes_ready,
                 bool multiply_adds = false) {
  Timer t(s);
  if (int e = factor_launch(w, n, precision, s, planes_ready, multiply_adds)) return e;
  return factor_finish(w, n, precision, info, s, t, multiply_adds);
}

int read_state(const SolveWs& w, int n, int* precision, bool* multiply_adds, cudaStream_t s) {
  int32_t state[kStateInts] = {};
  UPDES_CUDA_TRY(cudaMemcpyAsync(state, w.state, sizeof state, cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  if (state[2] != 1 || state[0] != n) return UPDES_ERR_INVALID;
  *precision = state[1];
  *multiply_adds = state[4] != 0;
  return UPDES_OK;
}

// K of a polyharmonic system in double-float (updes_assemble_df) with the power-of-two equilibration of the
// FP64 path: row maxima from the assembly, column maxima of the row-scaled hi plane, both planes scaled in
// place.  UNSUPPORTED when an entry falls outside the range in which double-float keeps its 48 bits (the
// caller then assembles in FP64).
int assemble_df_stage(const updes_problem* p, const SolveWs& w, int n, cudaStream_t s) {
  unsigned* rowmax = reinterpret_cast<unsigned*>(w.dc);  // float bits, then the column maxima, then dc
  int32_t* flag = reinterpret_cast<int32_t*>(w.r);       // free until the refinement
  UPDES_CUDA_TRY(cudaMemsetAsync(rowmax, 0, size_t(n) * sizeof(unsigned), s));
  UPDES_CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(int32_t), s));
  // the FP64 working matrix is free until the factorisation: the assembly's row records and coordinates
  int e = updes_assemble_df(p, w.Khi, w.Klo, w.ld, rowmax, flag, w.W, size_t(n) * w.ld * sizeof(double), s);
  if (e) return e;
  row_scale_bits_kernel<<<unsigned(ceil_div(n, 256)), 256, 0, s>>>(rowmax, n, w.dr);
  UPDES_LAUNCH_CHECK();
  UPDES_CUDA_TRY(cudaMemsetAsync(w.dc, 0, size_t(n) * sizeof(double), s));
  col_max_f32_kernel<<<dim3(unsigned(ceil_div(n, 256)), kColScaleChunks), 256, 0, s>>>(
      w.Khi, w.ld, n, w.dr, reinterpret_cast<unsigned long long*>(w.dc));
  UPDES_LAUNCH_CHECK();
  col_scale_kernel<<<unsigned(ceil_div(n, 256)), 256, 0, s>>>(n, w.dc);
  UPDES_LAUNCH_CHECK();
  {
    StatScope sc(kStatOther, s, 0.0, double(n) * n * 24.0);
    // the factorisation's working copy (F32, Wlo) in the same pass: the assembly's scratch there is done with
    scale_planes_kernel<<<dim3(unsigned(ceil_div(n, 1024)), unsigned(std::min(n, 4096))), 256, 0, s>>>(
        w.Khi, w.Klo, w.ld, n, w.dr, w.dc, w.F32, w.Wlo);
    UPDES_LAUNCH_CHECK();
  }
  int32_t hflag = 0;
  UPDES_CUDA_TRY(cudaMemcpyAsync(&hflag, flag, sizeof hflag, cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  return hflag ? UPDES_ERR_UNSUPPORTED : UPDES_OK;
}

// Assemble K and its power-of-two equilibration into the double-float planes: in double-float arithmetic for
// a polyharmonic system factored in FP32, else in FP64.
// *planes_ready: the factorisation's working copy holds the equilibrated K as well (the planes of a
// double-float assembly, or the FP64 K of an FP64 solve).
int assemble_stage(const updes_problem* p, const SolveWs& w, int n, int precision, updes_solve_info* info,
                   cudaStream_t s, bool* planes_ready) {
  Timer t(s);
  int e;
  *planes_ready = false;
  // UPDES_DF_ASSEMBLY=0 assembles every system in FP64
  static const bool df_assembly = [] {
    const char* v = std::getenv("UPDES_DF_ASSEMBLY");
    return !(v && v[0] == '0');
  }();
  if (df_assembly && precision == UPDES_PREC_FP32 && p->rbf == UPDES_RBF_POLYHARMONIC) {
    e = assemble_df_stage(p, w, n, s);
    if (e != UPDES_ERR_UNSUPPORTED) {
      if (e) return e;
      *planes_ready = true;
      info->t_assemble_ms += t.stop();
      return UPDES_OK;
    }
  }
  if ((e = updes_assemble(p, w.W, w.ld, nullptr, 0, s))) return e;  // FP64 K, staged in the working buffer
  // the mixed path by whole rows and columns, like its double-float assembly; the FP64 path over the kernel block first
  const int first = precision == UPDES_PREC_FP64 ? p->N : n;
  auto rows_by = [&](int rows, const double* dc) -> int {
    row_scale_kernel<<<unsigned(ceil_div(int64_t(rows) * 32, 256)), 256, 0, s>>>(w.W, w.ld, n, rows, rows, dc, w.dr);
    UPDES_LAUNCH_CHECK();
    return UPDES_OK;
  };
  auto columns_by = [&](int rows) -> int {
    UPDES_CUDA_TRY(cudaMemsetAsync(w.dc, 0, size_t(n) * sizeof(double), s));
    column_exponents_kernel<<<dim3(unsigned(ceil_div(n, 256)), kColScaleChunks), 256, 0, s>>>(
        w.W, w.ld, n, rows, w.dr, reinterpret_cast<int2*>(w.dc));
    UPDES_LAUNCH_CHECK();
    column_scale_kernel<<<unsigned(ceil_div(n, 256)), 256, 0, s>>>(n, w.dc);
    UPDES_LAUNCH_CHECK();
    return UPDES_OK;
  };
  if ((e = rows_by(first, nullptr)) || (e = columns_by(first))) return e;
  if (first < n) {
    polynomial_scale_kernel<<<2, 256, 0, s>>>(w.W, w.ld, first, n - first, w.dr, w.dc);
    UPDES_LAUNCH_CHECK();
    if ((e = rows_by(n, w.dc)) || (e = columns_by(n))) return e;
  }
  // the FP64 path factors the equilibrated FP64 K itself (written back in place), not the 48-bit sum of its
  // planes: on systems near the FP64 limit (r^5 at N = 10,000) the planes' rounding alone would be 32x the
  // FP64 rounding of K
  const int fp64 = precision == UPDES_PREC_FP64;
  split_df_kernel<<<unsigned(ceil_div(int64_t(n) * w.ld, 256)), 256, 0, s>>>(w.W, w.ld, w.Khi, w.Klo, w.ld, n, w.dr,
                                                                             w.dc, fp64);
  UPDES_LAUNCH_CHECK();
  *planes_ready = fp64 != 0;  // for the FP64 factorisation: W holds the equilibrated K
  info->t_assemble_ms += t.stop();
  return UPDES_OK;
}

// One right-hand side against the stored factors: refinement, FP64 fallback, coeffs and vals.
int solve_stage(const updes_problem* p, const SolveWs& w, int n, const double* q, int64_t qstride, double* coeffs,
                int64_t cstride, double* vals, int64_t vstride, const updes_solve_opts& o, updes_solve_info* info,
                cudaStream_t s) {
  const unsigned g = unsigned(ceil_div(n, 256));
  int precision, e;
  bool multiply_adds;
  if ((e = read_state(w, n, &precision, &multiply_adds, s))) return e;
  for (;;) {
    Timer t(s);
    if (qstride == 1) {
      rhs_kernel<<<g, 256, 0, s>>>(q, p->N, n, w.dr, w.bs);
      UPDES_LAUNCH_CHECK();
    } else {
      UPDES_CUDA_TRY(cudaMemsetAsync(w.r, 0, size_t(n) * 8, s));
      UPDES_CUDA_TRY(cudaMemcpy2DAsync(w.r, 8, q, qstride * 8, 8, p->N, cudaMemcpyDeviceToDevice, s));
      rhs_kernel<<<g, 256, 0, s>>>(w.r, p->N, n, w.dr, w.bs);
      UPDES_LAUNCH_CHECK();
    }
    abs_kernel<<<g, 256, 0, s>>>(w.bs, w.bsabs, n);
    UPDES_LAUNCH_CHECK();
    if ((e = precond(w, n, precision, w.bs, w.x, s))) return e;
    updes_solve_opts oi = o;
    if (precision == UPDES_PREC_FP64) oi.max_iters = 0;  // plain FP64 LU: report the residual only
    if ((e = gmres(w, n, precision, oi, info, s))) return e;
    DeviceStatus h;
    if ((e = read_status(w.lu.st, s, &h))) return e;
    if (h.error) return h.error;
    info->t_refine_ms += t.stop();
    bool again = precision == UPDES_PREC_FP64 && !multiply_adds && !info->lu_info;
    if (again && (e = digits_failed(w, n, false, *info, &again, s))) return e;
    if (precision == UPDES_PREC_FP64 && !again) {
      info->converged = 1;
      break;
    }
    if (precision == UPDES_PREC_FP32) {
      if (info->converged || !o.fallback_fp64) break;
      info->fell_back = 1;
    }
    precision = UPDES_PREC_FP64;
    multiply_adds = again;
    // the factors overwrote the working matrix, and the mixed path scales K in its own way: assembled and scaled again
    bool ready = false;
    if ((e = assemble_stage(p, w, n, precision, info, s, &ready))) return e;
    if ((e = factor_stage(w, n, precision, info, s, ready, multiply_adds))) return e;
  }
  Timer t(s);
  // the values of a mixed-precision solve in double-float (polyharmonic kernels; UPDES_DF_EVAL=0: FP64)
  static const bool df_eval_on = [] {
    const char* v = std::getenv("UPDES_DF_EVAL");
    return !(v && v[0] == '0');
  }();
  const bool df_eval = df_eval_on && precision == UPDES_PREC_FP32;
  axpby_kernel<<<g, 256, 0, s>>>(w.x, 1.0, w.x, 0.0, n, w.dc);  // coeffs = dc .* x
  UPDES_LAUNCH_CHECK();
  if (cstride == 1) {
    UPDES_CUDA_TRY(cudaMemcpyAsync(coeffs, w.x, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
    if (vals && vstride == 1 && (e = eval_values_sym(p, coeffs, vals, w.evp, s, df_eval))) return e;
  } else {
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(coeffs, cstride * 8, w.x, 8, 8, n, cudaMemcpyDeviceToDevice, s));
  }
  if (vals && (cstride != 1 || vstride != 1)) {
    if ((e = eval_values_sym(p, w.x, w.wv, w.evp, s, df_eval))) return e;
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(vals, vstride * 8, w.wv, 8, 8, p->N, cudaMemcpyDeviceToDevice, s));
  }
  info->t_eval_ms += t.stop();
  return UPDES_OK;
}

int solve_setup(const updes_problem* p, const updes_solve_opts* opts, void* workspace, size_t workspace_bytes,
                SolveWs* w, updes_solve_opts* o) {
  if (updes_check_problem(p) || !workspace) return UPDES_ERR_INVALID;
  *o = normalise(opts);
  if (o->precision != UPDES_PREC_FP64 && o->precision != UPDES_PREC_FP32) return UPDES_ERR_INVALID;
  const int n = p->N + p->M;
  updes_solve_opts olay = *o;
  olay.precision = UPDES_PREC_FP32;
  if (workspace_bytes < solve_ws_layout(n, olay, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  solve_ws_layout(n, olay, static_cast<char*>(workspace), w);
  return UPDES_OK;
}

}  // namespace

extern "C" int updes_factor(const updes_problem* p, const updes_solve_opts* opts, updes_solve_info* info,
                            void* workspace, size_t workspace_bytes, void* stream) {
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, opts, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  updes_solve_info dummy;
  if (!info) info = &dummy;
  std::memset(info, 0, sizeof *info);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = p->N + p->M;
  bool planes_ready = false;
  if ((e = assemble_stage(p, w, n, o.precision, info, s, &planes_ready))) return e;
  if ((e = factor_stage(w, n, o.precision, info, s, planes_ready))) return e;
  return info->lu_info ? UPDES_ERR_SINGULAR : UPDES_OK;
}

extern "C" int updes_solve_factored(const updes_problem* p, int32_t nrhs, const double* Q, int64_t ldq,
                                    double* coeffs, int64_t ldc, double* vals, int64_t ldv,
                                    const updes_solve_opts* opts, updes_solve_info* info, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, opts, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  if (nrhs <= 0 || !Q || !coeffs || ldq < nrhs || ldc < nrhs || (vals && ldv < nrhs)) return UPDES_ERR_INVALID;
  updes_solve_info dummy;
  if (!info) info = &dummy;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = p->N + p->M;
  updes_solve_info agg;
  std::memset(&agg, 0, sizeof agg);
  agg.converged = 1;
  for (int j = 0; j < nrhs; ++j) {
    updes_solve_info one;
    std::memset(&one, 0, sizeof one);
    if ((e = solve_stage(p, w, n, Q + j, ldq, coeffs + j, ldc, vals ? vals + j : nullptr, ldv, o, &one, s))) return e;
    agg.iters += one.iters;
    agg.fell_back |= one.fell_back;
    agg.lu_info = one.lu_info ? one.lu_info : agg.lu_info;
    agg.converged &= one.converged;
    agg.rel_residual = std::fmax(agg.rel_residual, one.rel_residual);
    agg.backward_error = std::fmax(agg.backward_error, one.backward_error);
    agg.t_factor_ms += one.t_factor_ms;
    agg.t_refine_ms += one.t_refine_ms;
    agg.t_eval_ms += one.t_eval_ms;
  }
  *info = agg;
  return agg.converged ? UPDES_OK : UPDES_ERR_NOT_CONVERGED;
}

namespace {
struct Pending {
  Timer t;
  updes_solve_info info;
  int n, precision;
};
}  // namespace

extern "C" int updes_solve_begin(const updes_problem* p, const updes_solve_opts* opts, void* workspace,
                                 size_t workspace_bytes, void* stream, void** pending) {
  SolveWs w;
  updes_solve_opts o;
  if (!pending) return UPDES_ERR_INVALID;
  *pending = nullptr;
  int e = solve_setup(p, opts, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = p->N + p->M;
  updes_solve_info info;
  std::memset(&info, 0, sizeof info);
  bool planes_ready = false;
  if ((e = assemble_stage(p, w, n, o.precision, &info, s, &planes_ready))) return e;
  std::unique_ptr<Pending> h(new (std::nothrow) Pending{Timer(s), info, n, o.precision});
  if (!h) return UPDES_ERR_CUDA;
  if ((e = factor_launch(w, n, o.precision, s, planes_ready))) return e;
  h->t.mark();
  *pending = h.release();
  return UPDES_OK;
}

extern "C" int updes_solve_end(void* pending, const updes_problem* p, const double* q, double* coeffs, double* vals,
                               const updes_solve_opts* opts, updes_solve_info* info, void* workspace,
                               size_t workspace_bytes, void* stream) {
  if (!pending) return UPDES_ERR_INVALID;
  std::unique_ptr<Pending> h(static_cast<Pending*>(pending));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!q) {  // given up: nothing of it runs any more when the call returns
    UPDES_CUDA_TRY(cudaStreamSynchronize(s));
    return UPDES_OK;
  }
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, opts, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  const int n = p->N + p->M;
  if (!coeffs || n != h->n || o.precision != h->precision) return UPDES_ERR_INVALID;
  updes_solve_info dummy;
  if (!info) info = &dummy;
  *info = h->info;
  if ((e = factor_finish(w, n, o.precision, info, s, h->t))) return e;
  if ((e = solve_stage(p, w, n, q, 1, coeffs, 1, vals, 1, o, info, s))) return e;
  if (info->lu_info) return UPDES_ERR_SINGULAR;
  if (!info->converged) return UPDES_ERR_NOT_CONVERGED;
  return UPDES_OK;
}

extern "C" int updes_solve(const updes_problem* p, const double* q, double* coeffs, double* vals,
                           const updes_solve_opts* opts, updes_solve_info* info, void* workspace,
                           size_t workspace_bytes, void* stream) {
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, opts, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  if (!q || !coeffs) return UPDES_ERR_INVALID;
  updes_solve_info dummy;
  if (!info) info = &dummy;
  std::memset(info, 0, sizeof *info);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = p->N + p->M;
  bool planes_ready = false;
  if ((e = assemble_stage(p, w, n, o.precision, info, s, &planes_ready))) return e;
  if ((e = factor_stage(w, n, o.precision, info, s, planes_ready))) return e;
  if ((e = solve_stage(p, w, n, q, 1, coeffs, 1, vals, 1, o, info, s))) return e;
  if (info->lu_info) return UPDES_ERR_SINGULAR;
  if (!info->converged) return UPDES_ERR_NOT_CONVERGED;
  return UPDES_OK;
}

// ---------------------------------------------------------------------------
// Triangular solves with a fixed, library-owned scratch (no allocation at all)
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoallocSyncOff = 256;                                   // after the status word
constexpr size_t kNoallocVecOff = 2304;                                   // after (n/64 + 2) flags
constexpr size_t kNoallocBytes = kNoallocVecOff + 2 * size_t(UPDES_NOALLOC_MAX_N) * sizeof(double);
static_assert(kNoallocVecOff - kNoallocSyncOff >= sizeof(int) * (UPDES_NOALLOC_MAX_N / 64 + 2), "flag region");

// The only scratch of updes_lu_solve_noalloc, shared by all its calls on a device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

std::mutex g_noalloc_mu;
constexpr int kMaxDevices = 64;
void* g_noalloc_addr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device (looked up once per device, by the first call
// there).  Devices with ordinal 64 or more are not supported; a lookup that fails while `s` is being captured
// says so, since that first call has to be made outside capture.
int noalloc_scratch(void** out, cudaStream_t s) {
  int dev = 0;
  UPDES_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    updes_set_last_cuda_error(cudaErrorInvalidDevice, "updes_lu_solve_noalloc supports device ordinals 0..63",
                              __FILE__, __LINE__);
    return UPDES_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      const bool capturing = cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
      updes_set_last_cuda_error(e, capturing ? "cudaGetSymbolAddress(g_noalloc_scratch) during stream capture: make "
                                               "the first updes_lu_solve_noalloc call on a device before any capture"
                                             : "cudaGetSymbolAddress(g_noalloc_scratch)",
                                __FILE__, __LINE__);
      return UPDES_ERR_CUDA;
    }
    g_noalloc_addr[dev] = p;
  }
  *out = g_noalloc_addr[dev];
  return UPDES_OK;
}

}  // namespace

extern "C" int updes_lu_solve_noalloc(int32_t n, const void* F, int64_t ldf, int32_t precision, const int32_t* piv,
                                      double* b, int32_t nrhs, int64_t ldb, int32_t trans, void* stream) {
  if (n <= 0 || !F || ldf < n || !piv || !b || nrhs <= 0 || ldb < nrhs) return UPDES_ERR_INVALID;
  if (precision != UPDES_PREC_FP64 && precision != UPDES_PREC_FP32) return UPDES_ERR_INVALID;
  if (n > UPDES_NOALLOC_MAX_N) return UPDES_ERR_TOO_LARGE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* base = nullptr;
  int e = noalloc_scratch(&base, s);
  if (e) return e;
  char* c = static_cast<char*>(base);
  LuWs w{};
  w.st = reinterpret_cast<DeviceStatus*>(c);
  w.sync = reinterpret_cast<int*>(c + kNoallocSyncOff);
  w.tmp = reinterpret_cast<double*>(c + kNoallocVecOff);
  double* col = w.tmp + UPDES_NOALLOC_MAX_N;
  UPDES_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(DeviceStatus), s));  // the flags are cleared by each solve
  for (int j = 0; j < nrhs; ++j) {
    double* bj = b + j;
    if (nrhs == 1) {
      if ((e = solve_any(n, F, ldf, precision, piv, bj, trans, w, s))) return e;
      continue;
    }
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(col, 8, bj, ldb * 8, 8, n, cudaMemcpyDeviceToDevice, s));
    if ((e = solve_any(n, F, ldf, precision, piv, col, trans, w, s))) return e;
    UPDES_CUDA_TRY(cudaMemcpy2DAsync(bj, ldb * 8, col, 8, 8, n, cudaMemcpyDeviceToDevice, s));
  }
  DeviceStatus h;
  if ((e = read_status(w.st, s, &h))) return e;
  return h.error;
}

// Views into a solve workspace (after updes_factor) for the batched solves.
int solve_ws_views(const updes_problem* p, void* workspace, size_t workspace_bytes, const float** Khi,
                   const float** Klo, const float** F32, const double** F64, int64_t* ld, const int32_t** piv,
                   const double** dr, const double** dc, DeviceStatus** st, const int32_t** state) {
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, nullptr, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  *Khi = w.Khi;
  *Klo = w.Klo;
  *F32 = w.F32;
  *F64 = w.W;
  *ld = w.ld;
  *piv = w.piv;
  *dr = w.dr;
  *dc = w.dc;
  *st = w.lu.st;
  *state = w.state;
  return UPDES_OK;
}

extern "C" int updes_workspace_status(const updes_problem* p, void* workspace, size_t workspace_bytes,
                                      int32_t* error, void* stream) {
  SolveWs w;
  updes_solve_opts o;
  int e = solve_setup(p, nullptr, workspace, workspace_bytes, &w, &o);
  if (e) return e;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DeviceStatus h;
  if ((e = read_status(w.lu.st, s, &h))) return e;
  if (error) *error = h.error;
  UPDES_CUDA_TRY(cudaMemsetAsync(w.lu.st, 0, sizeof(DeviceStatus), s));
  return UPDES_OK;
}

// ---------------------------------------------------------------------------
// Adjoint: K^T lambda = g with the factors left in the workspace by updes_solve
// ---------------------------------------------------------------------------
extern "C" int updes_solve_transpose(const updes_problem* p, const double* g, double* lambda,
                                     const updes_solve_opts* opts, updes_solve_info* info, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  if (updes_check_problem(p) || !g || !lambda || !workspace) return UPDES_ERR_INVALID;
  updes_solve_opts o = normalise(opts);
  const int n = p->N + p->M;
  updes_solve_opts olay = o;
  olay.precision = UPDES_PREC_FP32;
  if (workspace_bytes < solve_ws_layout(n, olay, nullptr, nullptr)) return UPDES_ERR_WORKSPACE;
  SolveWs w;
  solve_ws_layout(n, olay, static_cast<char*>(workspace), &w);
  updes_solve_info dummy;
  if (!info) info = &dummy;
  std::memset(info, 0, sizeof *info);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int precision = 0, e;
  bool multiply_adds;
  if ((e = read_state(w, n, &precision, &multiply_adds, s))) return e;  // no factorisation of this system in the workspace
  const unsigned gr = unsigned(ceil_div(n, 256));
  Timer t(s);
  for (;;) {
    UPDES_CUDA_TRY(cudaMemsetAsync(w.lu.st, 0, sizeof(DeviceStatus), s));
    // K^T lambda = g  <=>  Ks^T mu = dc .* g,  lambda = dr .* mu
    UPDES_CUDA_TRY(cudaMemcpyAsync(w.bs, g, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
    axpby_kernel<<<gr, 256, 0, s>>>(w.bs, 1.0, w.bs, 0.0, n, w.dc);
    UPDES_LAUNCH_CHECK();
    abs_kernel<<<gr, 256, 0, s>>>(w.bs, w.bsabs, n);
    UPDES_LAUNCH_CHECK();
    UPDES_CUDA_TRY(cudaMemcpyAsync(w.x, w.bs, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
    if ((e = precond(w, n, precision, w.x, w.x, s, true))) return e;
    updes_solve_opts oi = o;
    if (precision == UPDES_PREC_FP64) oi.max_iters = 0;
    if ((e = gmres(w, n, precision, oi, info, s, true))) return e;
    if (precision != UPDES_PREC_FP64 || multiply_adds) break;
    if ((e = digits_failed(w, n, true, *info, &multiply_adds, s))) return e;
    if (!multiply_adds) break;
    bool ready = false;
    if ((e = assemble_stage(p, w, n, precision, info, s, &ready))) return e;
    if ((e = factor_stage(w, n, precision, info, s, ready, multiply_adds))) return e;
  }
  if (precision == UPDES_PREC_FP64) info->converged = 1;
  info->fell_back = precision == UPDES_PREC_FP64 && o.precision == UPDES_PREC_FP32;
  axpby_kernel<<<gr, 256, 0, s>>>(w.x, 1.0, w.x, 0.0, n, w.dr);
  UPDES_LAUNCH_CHECK();
  UPDES_CUDA_TRY(cudaMemcpyAsync(lambda, w.x, size_t(n) * 8, cudaMemcpyDeviceToDevice, s));
  DeviceStatus h;
  if ((e = read_status(w.lu.st, s, &h))) return e;
  if (h.error) return h.error;
  info->t_refine_ms = t.stop();
  return info->converged ? UPDES_OK : UPDES_ERR_NOT_CONVERGED;
}
