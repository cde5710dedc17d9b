// Many independent collocation systems of uneven size in ONE persistent launch (updes_solve_batched).
//
// The reference solves each system with its own pde_solver call (updes/operators.py:559-618).  Systems of a
// few hundred to a few thousand nodes leave most of a GB300 idle one at a time, and a solve made of hundreds
// of small launches per system is bound by launch and synchronisation latency.  Here CTAs (one per SM), and for the
// largest systems thread-block clusters of eight, take systems from device work queues (largest first) and run the
// whole solve of each by themselves:
//
//   assembly   K (FP64, closed forms of entries.cuh), equilibrated by powers of two (rows, then columns);
//              the value matrix A[:N] = [Phi P] for vals, in FP64
//   LU         right-looking, partial pivoting (LAPACK's pivot rule), panel width nb chosen per system size
//              by the autotuner (updes_batched_tune); the elimination in double-float arithmetic on the FP32
//              pipes (UPDES_PREC_FP32: about 48-bit factors, GB300's FP64 pipe is 1/64 of its FP32 rate) or
//              in FP64 (UPDES_PREC_FP64)
//   refinement y = (LU)^-1 b, then classical refinement sweeps y += (LU)^-1 (b - K y) with an FP64 residual
//              while the componentwise backward error still halves (down to 2 FP64 unit roundoffs; 32
//              count as converged) and the sweep cap is not met; with 48-bit factors each sweep gains a factor of about 1 / (cond(K) 2^-48),
//              so one or two sweeps reach the floor wherever cond(K) 2^-48 is small
//   values     coeffs = Dc y, vals = A[:N] coeffs
//
// The scratch of a CTA or cluster (its slice of the workspace) holds K, the working matrix and A for the largest
// system.  Every wait is a CTA or cluster barrier (the CTAs of a cluster run at the same time), so nothing can hang.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <new>
#include <numeric>
#include <queue>
#include <vector>

#include "common.cuh"
#include "df.cuh"
#include "entries.cuh"
#include "rbf.cuh"
#include "side_stream.cuh"
#include "stats.cuh"

int updes_check_problem(const updes_problem* p);

namespace {

constexpr int kBT = 512;                 // threads per CTA
constexpr int kWarps = kBT / 32;
constexpr int kTM = 64, kTN = 64;        // trailing-update tile of half a CTA: 4 x 4 entries per thread
constexpr int kTeams = 2;                // half CTAs, each on tiles of its own: one computes while the other loads
constexpr int kMaxNB = 64;               // widest panel
constexpr int kCoopNB = 32;              // panel width of a cluster: its panels are short chains whatever their width,
                                         // and wider panels read the trailing matrix less often
constexpr int kMaxBatchN = 4096;         // the solve's vectors live in shared memory
constexpr int kMaxC = 8;                 // CTAs of a cooperative solve
// A solve counts as converged at a componentwise backward error of 32 FP64 unit roundoffs (the residual is
// FP64 here, K being kept in FP64), but refinement goes on while the error still halves, down to 2 unit
// roundoffs: on the r^5 systems of a few hundred nodes the vals only agree with an FP64 LU's to within
// FP64's own spread once the backward error is a few unit roundoffs.
constexpr double kBwdFloorB = 32.0 * 1.1102230246251565e-16;
constexpr double kBwdStop = 2.0 * 1.1102230246251565e-16;

struct BatchSys {
  updes_problem p;
  const double* q;
  double* coeffs;
  double* vals;
  int32_t n, nb, precision, max_sweeps;
};

struct BatchOut {
  int32_t lu_info, sweeps, converged, done;
  double backward_error;
};

// Shared memory of one CTA: a panel's rows, or the update's staged tiles, or the solve's two vectors and a staged block.
struct TeamTiles {
  float4 L[kTM][kMaxNB];  // L21 rows of the current row chunk: the elimination's stage_l writes and reads them
  double U[kMaxNB][kTN];  // U12 columns of the current column chunk (stage_u)
};
union SmemLU {
  TeamTiles team[kTeams];
  double L11[kMaxNB][kMaxNB];  // unit lower diagonal block of the panel
};
constexpr size_t kSmemBytes = 204 * 1024;
static_assert(sizeof(SmemLU) <= kSmemBytes && 2 * kMaxBatchN * sizeof(double) + 32 * 33 * 8 <= kSmemBytes, "shared memory");

// The rows of a panel column's exchange.
struct PanelRows {
  double cand[2][kMaxNB];  // by column parity: this CTA's best row, and the row at the diagonal if it has it
  double diag[2][kMaxNB];
  double prow[kMaxNB], drow[kMaxNB];
  double inv;              // 1 / pivot in the elimination's type, 0 for an unusable pivot
  int ok;
  int piv[kMaxNB];
  int start[kMaxC + 1];    // first row of every CTA's run
};

// Element arithmetic of the elimination: FP64, or double-float (F2, 8 bytes like a double).
struct OpsF64 {
  using T = double;
  static __device__ __forceinline__ T from_d(double v) { return v; }
  static __device__ __forceinline__ double to_d(T a) { return a; }
  static __device__ __forceinline__ void fms(T& c, T a, T b) { c = fma(-a, b, c); }  // c -= a b
  static __device__ __forceinline__ T mul(T a, T b) { return a * b; }
  // column b (of 4) of thread tc's entries in a tile: a warp's loads of a U row are 16 consecutive entries
  static __device__ __forceinline__ int column(int tc, int b) { return tc + 16 * b; }
  static __device__ __forceinline__ void stage_l(TeamTiles& s, int r, int k, T v) {
    reinterpret_cast<T*>(s.L)[r * kMaxNB + k] = v;
  }
  static __device__ __forceinline__ void stage_u(TeamTiles& s, int k, int c, T v) { s.U[k][c] = v; }
  // acc[a][b] -= sum_k L[row + a][k] U[k][column(tc, b)]
  static __device__ __forceinline__ void tile_update(T (&acc)[4][4], const TeamTiles& s, int row, int tc, int kb) {
    const T* L = reinterpret_cast<const T*>(s.L) + row * kMaxNB;
    for (int k = 0; k < kb; ++k) {
      T la[4], ub[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) la[a] = L[a * kMaxNB + k];
#pragma unroll
      for (int b = 0; b < 4; ++b) ub[b] = s.U[k][column(tc, b)];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) fms(acc[a][b], la[a], ub[b]);
    }
  }
};

struct OpsDF {
  using T = F2;
  static __device__ __forceinline__ T from_d(double v) { return df_from_double(v); }
  static __device__ __forceinline__ double to_d(T a) { return double(a.h) + double(a.l); }
  // c -= a b: the exact product of the high parts by FMA plus the cross terms, subtracted by TwoSum, then
  // renormalised (every operation an _rn intrinsic, so the compiler cannot contract the error terms away)
  static __device__ __forceinline__ void fms(T& c, T a, T b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, e));
    const float s = __fsub_rn(c.h, p);
    const float v = __fsub_rn(s, c.h);
    float t = __fsub_rn(__fsub_rn(c.h, __fsub_rn(s, v)), __fadd_rn(p, v));
    t = __fadd_rn(t, __fsub_rn(c.l, e));
    const float h = __fadd_rn(s, t);
    c.l = __fsub_rn(t, __fsub_rn(h, s));
    c.h = h;
  }
  static __device__ __forceinline__ T mul(T a, T b) { return df_mul(a, b); }
  // fms on two columns at once with the packed FP32x2 instructions of sm_100+: the same operations, with -a b as the
  // product of -a (rounding is symmetric) so that nothing is negated, hence bitwise the same results; y - x is
  // fma(x, -1, y), which rounds once like the subtraction.  A packed instruction takes the FMA pipe two cycles, and so
  // does every move that puts a pair together: the tiles are staged as the pairs that are read, an L entry as
  // (h, h, l, l), a row of U as a plane of high and one of low parts (the moves took 40 % of the pipe).
  static __device__ __forceinline__ float2 sub2(float2 y, float2 x) {
    return __ffma2_rn(x, make_float2(-1.f, -1.f), y);
  }
  static __device__ __forceinline__ void fms2(float2& ch, float2& cl, float2 ah, float2 nah, float2 al, float2 bh,
                                              float2 bl) {
    const float2 np = __fmul2_rn(nah, bh);
    float2 e = __ffma2_rn(ah, bh, np);
    e = __ffma2_rn(ah, bl, __ffma2_rn(al, bh, e));
    const float2 s = __fadd2_rn(ch, np);
    const float2 v = sub2(s, ch);
    float2 t = __fadd2_rn(sub2(ch, sub2(s, v)), sub2(np, v));
    t = __fadd2_rn(t, sub2(cl, e));
    const float2 h = __fadd2_rn(s, t);
    cl = sub2(t, sub2(h, s));
    ch = h;
  }
  static __device__ __forceinline__ int column(int tc, int b) { return 2 * tc + (b & 1) + 32 * (b >> 1); }
  static __device__ __forceinline__ void stage_l(TeamTiles& s, int r, int k, T v) {
    s.L[r][k] = make_float4(v.h, v.h, v.l, v.l);
  }
  static __device__ __forceinline__ void stage_u(TeamTiles& s, int k, int c, T v) {
    float* u = reinterpret_cast<float*>(s.U);
    u[k * kTN + c] = v.h;
    u[(kMaxNB + k) * kTN + c] = v.l;
  }
  static __device__ __forceinline__ void tile_update(T (&acc)[4][4], const TeamTiles& s, int row, int tc, int kb) {
    float2 ch[4][2], cl[4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        ch[a][q] = make_float2(acc[a][2 * q].h, acc[a][2 * q + 1].h);
        cl[a][q] = make_float2(acc[a][2 * q].l, acc[a][2 * q + 1].l);
      }
    const float* u = reinterpret_cast<const float*>(s.U) + 2 * tc;
    for (int k = 0; k < kb; ++k) {
      float2 bh[2], bl[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        bh[q] = *reinterpret_cast<const float2*>(u + k * kTN + 32 * q);
        bl[q] = *reinterpret_cast<const float2*>(u + (kMaxNB + k) * kTN + 32 * q);
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float4 l = s.L[row + a][k];
        const float2 ah = make_float2(l.x, l.y), al = make_float2(l.z, l.w);
        const float2 nah = make_float2(__uint_as_float(__float_as_uint(l.x) ^ 0x80000000u),
                                       __uint_as_float(__float_as_uint(l.y) ^ 0x80000000u));
#pragma unroll
        for (int q = 0; q < 2; ++q) fms2(ch[a][q], cl[a][q], ah, nah, al, bh[q], bl[q]);
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        acc[a][2 * q] = {ch[a][q].x, cl[a][q].x};
        acc[a][2 * q + 1] = {ch[a][q].y, cl[a][q].y};
      }
  }
};

__device__ __forceinline__ double pow2_scale(double m) {
  // 2^-e with m = f 2^e, f in [0.5, 1): scales m into [0.5, 1) exactly; 1 for m = 0 or non-finite m
  int e = 0;
  if (m > 0.0 && isfinite(m)) frexp(m, &e);
  return ldexp(1.0, -e);
}

// The CTAs that solve one system: a thread-block cluster (COOP), whose threads share the rows, columns and tiles of
// every phase, or one CTA by itself.  Either way each entry sees the same operations in the same order, so the results
// are bitwise the same.
struct Exchange {
  double v[2][kMaxC];
  int i[2][kMaxC];
};

template <bool COOP>
struct Group {
  int rank = 0, ctas = 1;
  int parity = 0;  // of the exchange slots: one is rewritten two barriers after it was read
  Exchange* ex = nullptr;
  __device__ __forceinline__ int thread() const { return COOP ? rank * kBT + int(threadIdx.x) : int(threadIdx.x); }
  __device__ __forceinline__ int threads() const { return COOP ? ctas * kBT : kBT; }
  __device__ __forceinline__ int warp() const { return thread() >> 5; }
  __device__ __forceinline__ int warps() const { return COOP ? ctas * kWarps : kWarps; }
  __device__ __forceinline__ void sync() const {
    if constexpr (COOP)
      asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
      __syncthreads();
  }
  // the address of one of this CTA's shared variables in CTA `cta` of the cluster
  static __device__ __forceinline__ uint32_t remote(const void* p, int cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(cta));
    return r;
  }
  static __device__ __forceinline__ void put(uint32_t at, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
  }
  // an 8-byte shared variable of CTA `cta`
  static __device__ __forceinline__ double get(const double* p, int cta) {
    if constexpr (!COOP) return *p;
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote(p, cta)) : "memory");
    return v;
  }
  // every CTA's (v, i) to every CTA (all threads hold the same pair); the group's largest v (none negative: compared by
  // their bits), smallest i on ties
  __device__ __forceinline__ void argmax(double& v, int& i) {
    if constexpr (COOP) {
      if (int(threadIdx.x) < ctas) {
        put(remote(&ex->v[parity][rank], int(threadIdx.x)), v);
        asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(remote(&ex->i[parity][rank], int(threadIdx.x))), "r"(i)
                     : "memory");
      }
      sync();
      unsigned long long k = static_cast<unsigned long long>(__double_as_longlong(ex->v[parity][0]));
      i = ex->i[parity][0];
      for (int c = 1; c < ctas; ++c) {
        const unsigned long long ok = static_cast<unsigned long long>(__double_as_longlong(ex->v[parity][c]));
        const int oi = ex->i[parity][c];
        if (ok > k || (ok == k && oi < i)) { k = ok; i = oi; }
      }
      v = __longlong_as_double(static_cast<long long>(k));
      parity ^= 1;
    }
  }
};

// Order key of a pivot candidate's |a|: its bits + 1, which order like the values (NaN counts as infinity, so it wins and
// surfaces as a bad pivot); 0 for no candidate.  Integers, because the FP64 pipe takes a comparison 64 cycles.
using Key = unsigned long long;
__device__ __forceinline__ Key key_of(double a) {
  return min(static_cast<Key>(__double_as_longlong(a)) & 0x7fffffffffffffffull, Key(0x7ff0000000000000ull)) + 1;
}
// The warp's largest key and the smallest row that has it.
__device__ __forceinline__ void warp_best(Key& key, int& row) {
  const unsigned hi = unsigned(key >> 32), lo = unsigned(key);
  const unsigned hm = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lm = __reduce_max_sync(0xffffffffu, hi == hm ? lo : 0u);
  row = __reduce_min_sync(0xffffffffu, (hi == hm && lo == lm) ? row : 0x7fffffff);
  key = (Key(hm) << 32) | lm;
}
// The group's best candidate from every thread's.
template <bool COOP>
__device__ __forceinline__ void group_best(Key& key, int& row, Key* red_k, int* red_i, Group<COOP>& grp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  warp_best(key, row);
  if (lane == 0) { red_k[w] = key; red_i[w] = row; }
  __syncthreads();
  key = red_k[lane & (kWarps - 1)];
  row = red_i[lane & (kWarps - 1)];
  warp_best(key, row);
}

__device__ __forceinline__ double cta_max(double v, double* red_v) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) red_v[w] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < kWarps; ++k) red_v[0] = fmax(red_v[0], red_v[k]);
  __syncthreads();
  v = red_v[0];
  __syncthreads();
  return v;
}

// ---- assembly ---------------------------------------------------------------------------------------------

// K (n x ld, FP64) and A[:N] (N x ld, FP64) of one system, K equilibrated in place: dr (rows) and dc
// (columns) are the powers of two applied, b = Dr [q; 0].  One warp per row.
template <int KIND, bool COOP>
__device__ void assemble_system(const BatchSys& sys, double* K, double* A, int64_t ld, double* dr, double* dc,
                                double* b, double* part, const Group<COOP>& grp) {
  const updes_problem& p = sys.p;
  const int n = sys.n, lane = threadIdx.x & 31;
  const int ip = (KIND == UPDES_RBF_POLYHARMONIC) ? 2 * int(p.rbf_param) + 1 : int(p.rbf_param);
  for (int r = grp.warp(); r < n; r += grp.warps()) {
    const RowInfo ri = load_row(p, r);
    double* Kr = K + int64_t(r) * ld;
    double* Ar = A + int64_t(r) * ld;
    // the value row of node r, A[r] = [phi(x_r - x_j) (0 at j = r), m_k(x_r)], from the same kernel
    // evaluations as K's row where the row's evaluation node is r
    const bool fused = r < p.N && ri.a == r;
    double mx = 0.0;
    for (int c = lane; c < n; c += 32) {
      double v;
      if (c < p.N) {
        const double xc = p.nodes[2ll * c], yc = p.nodes[2ll * c + 1];
        if (fused) {
          double phi;
          v = entry_rbf_phi<KIND>(ri, c, xc, yc, p.rbf_param, ip, p.self_term, &phi);
          Ar[c] = phi;
        } else {
          v = entry_rbf<KIND>(ri, c, xc, yc, p.rbf_param, ip, p.self_term);
        }
      } else {
        v = entry_mono(ri, c - p.N);
      }
      Kr[c] = v;
      mx = fmax(mx, fabs(v));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const double s = pow2_scale(mx);
    for (int c = lane; c < n; c += 32) Kr[c] *= s;
    if (lane == 0) {
      dr[r] = s;
      b[r] = r < p.N ? s * sys.q[r] : 0.0;
    }
    if (r < p.N) {
      const double xr = p.nodes[2ll * r], yr = p.nodes[2ll * r + 1];
      for (int c = lane; c < n; c += 32) {
        if (c >= p.N) Ar[c] = monomial_terms(c - p.N, xr, yr).m;
        else if (!fused)
          Ar[c] = (c == r && !p.self_term) ? 0.0 : rbf_value<KIND>(xr - p.nodes[2ll * c], yr - p.nodes[2ll * c + 1], p.rbf_param, ip);
      }
    }
  }
  grp.sync();
  // column powers of two over the row-scaled K: a CTA takes a range of rows (a maximum does not depend on the order)
  const int r0 = int(int64_t(n) * grp.rank / grp.ctas), r1 = int(int64_t(n) * (grp.rank + 1) / grp.ctas);
  for (int c = threadIdx.x; c < n; c += kBT) {
    double mx = 0.0;
#pragma unroll 8
    for (int r = r0; r < r1; ++r) mx = fmax(mx, fabs(K[int64_t(r) * ld + c]));
    if constexpr (COOP) part[int64_t(grp.rank) * n + c] = mx;
    else dc[c] = pow2_scale(mx);
  }
  grp.sync();
  if constexpr (COOP) {
    for (int c = grp.thread(); c < n; c += grp.threads()) {
      double mx = 0.0;
      for (int k = 0; k < grp.ctas; ++k) mx = fmax(mx, part[int64_t(k) * n + c]);
      dc[c] = pow2_scale(mx);
    }
    grp.sync();
  }
}

// W = K (scaled) converted to the elimination's type.
template <class Ops, bool COOP>
__device__ void scale_columns_to_w(const BatchSys& sys, double* K, typename Ops::T* W, int64_t ld, const double* dc,
                                   const Group<COOP>& grp) {
  const int n = sys.n;
  for (int r = grp.warp(); r < n; r += grp.warps()) {
    double* Kr = K + int64_t(r) * ld;
    typename Ops::T* Wr = W + int64_t(r) * ld;
    for (int c = threadIdx.x & 31; c < n; c += 32) {
      const double v = Kr[c] * dc[c];
      Kr[c] = v;
      Wr[c] = Ops::from_d(v);
    }
  }
  grp.sync();
}

// ---- LU -----------------------------------------------------------------------------------------------------

// Panel [k0, k0 + kb) of the rows [k0, n), in shared memory: the group's CTAs hold consecutive runs of rows.  Per
// column: CTA maximum (taken while the column was updated), the best row and the diagonal row staged, one cluster
// barrier, the winner's row and the diagonal row fetched, the interchange and the update of the CTA's own rows, a
// thread per row.  The interchanges of the columns outside the panel follow at its end, a thread per column.
// (With the rows in global memory, a row per thread, and every interchange at once a column took 15 to 20 us on eight
// CTAs, this about 3.)
template <class Ops, bool COOP>
__device__ int group_panel(typename Ops::T* W, int64_t ld, int n, int k0, int kb, int32_t* piv, SmemLU& sm,
                           PanelRows& pr, Key* red_k, int* red_i, Group<COOP>& grp) {
  using T = typename Ops::T;
  static_assert(sizeof(T) == 8, "rows travel as 8-byte words");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = n - k0, ldt = kb | 1;
  if (tid <= grp.ctas) pr.start[tid] = k0 + int(int64_t(m) * tid / grp.ctas);
  __syncthreads();
  const int rlo = pr.start[grp.rank], rows = pr.start[grp.rank + 1] - rlo;
  T* tile = reinterpret_cast<T*>(&sm);
  T* prow = reinterpret_cast<T*>(pr.prow);
  T* drow = reinterpret_cast<T*>(pr.drow);
  for (int l = warp; l < rows; l += kWarps)
    for (int c = lane; c < kb; c += 32) tile[l * ldt + c] = W[int64_t(rlo + l) * ld + k0 + c];
  __syncthreads();
  int info = 0;
  Key bk = 0;
  int bi = n;
  auto candidate = [&](T x, int row) {
    const Key k = key_of(Ops::to_d(x));
    if (k > bk) { bk = k; bi = row; }
  };
  for (int l = tid; l < rows; l += kBT) candidate(tile[l * ldt], rlo + l);
  for (int j = 0; j < kb; ++j) {
    const int par = j & 1, dg = k0 + j;
    group_best(bk, bi, red_k, red_i, grp);
    if (tid < kb && bi >= rlo && bi < rlo + rows)
      reinterpret_cast<T*>(pr.cand[par])[tid] = tile[(bi - rlo) * ldt + tid];
    if (tid >= 64 && tid - 64 < kb && dg >= rlo && dg < rlo + rows)
      reinterpret_cast<T*>(pr.diag[par])[tid - 64] = tile[(dg - rlo) * ldt + tid - 64];
    if constexpr (COOP) {
      double v = __longlong_as_double(static_cast<long long>(bk));  // (a key travels and compares as its bits)
      grp.argmax(v, bi);
    } else {
      __syncthreads();
    }
    const int p = bi < n ? bi : dg;
    if (tid < 128 && (tid & 63) < kb) {
      // the owner of row r: the last CTA whose run starts at or before it
      const int c = tid & 63, r = tid < 64 ? p : dg;
      int owner = 0;
      for (int q = 1; q < grp.ctas; ++q)
        if (pr.start[q] <= r) owner = q;
      const double* from = tid < 64 ? (bi < n ? pr.cand[par] : pr.diag[par]) : pr.diag[par];
      (tid < 64 ? pr.prow : pr.drow)[c] = Group<COOP>::get(from + c, owner);
      if (tid == j) {  // one thread's division, while the rows are interchanged
        const double pv = Ops::to_d(prow[j]);
        const bool ok = pv != 0.0 && isfinite(pv);
        reinterpret_cast<T&>(pr.inv) = Ops::from_d(ok ? 1.0 / pv : 0.0);
        pr.ok = ok;
        pr.piv[j] = p;
      }
    }
    __syncthreads();
    if (p != dg) {  // the interchange inside the panel
      if (tid < kb && dg >= rlo && dg < rlo + rows) tile[(dg - rlo) * ldt + tid] = prow[tid];
      if (tid >= 64 && tid - 64 < kb && p >= rlo && p < rlo + rows) tile[(p - rlo) * ldt + tid - 64] = drow[tid - 64];
    }
    __syncthreads();
    bk = 0;
    bi = n;
    const T inv = reinterpret_cast<const T&>(pr.inv);
    const bool ok = pr.ok;
    if (tid == 0 && !ok && info == 0) info = dg + 1;
    for (int l = max(0, dg + 1 - rlo) + tid; l < rows; l += kBT) {
      T* row = tile + l * ldt;
      if (ok) {
        const T x = Ops::mul(row[j], inv);
        row[j] = x;
        for (int c = j + 1; c < kb; ++c) Ops::fms(row[c], x, prow[c]);
      }
      if (j + 1 < kb) candidate(row[j + 1], rlo + l);
    }
  }
  __syncthreads();
  for (int l = warp; l < rows; l += kWarps)
    for (int c = lane; c < kb; c += 32) W[int64_t(rlo + l) * ld + k0 + c] = tile[l * ldt + c];
  if (grp.rank == 0 && tid < kb) piv[k0 + tid] = pr.piv[tid];
  for (int c0 = grp.thread(); c0 < n - kb; c0 += grp.threads()) {
    T* col = W + (c0 < k0 ? c0 : c0 + kb);
    for (int j = 0; j < kb; ++j) {
      const int p = pr.piv[j];
      if (p != k0 + j) {
        const T a = col[int64_t(k0 + j) * ld], b = col[int64_t(p) * ld];
        col[int64_t(k0 + j) * ld] = b;
        col[int64_t(p) * ld] = a;
      }
    }
  }
  grp.sync();
  return info;
}

template <class Ops, bool COOP>
__device__ int group_lu(typename Ops::T* W, int64_t ld, int n, int nb_max, int32_t* piv, SmemLU& sm, PanelRows& pr,
                        Key* red_k, int* red_i, Group<COOP>& grp) {
  using T = typename Ops::T;
  const int tid = threadIdx.x, team = tid / (kBT / kTeams), ttid = tid % (kBT / kTeams);
  int info = 0;
  TeamTiles& tiles_s = sm.team[team];
  T* L11 = reinterpret_cast<T*>(&sm.L11[0][0]);
  auto team_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(kBT / kTeams) : "memory"); };
  int kb;
  for (int k0 = 0; k0 < n; k0 += kb) {
    // the widest panel whose rows fit in shared memory (an entry's operations do not depend on the width)
    const int rows = (n - k0 + grp.ctas - 1) / grp.ctas;
    kb = min(nb_max, n - k0);
    while (size_t(rows) * (kb | 1) * sizeof(T) > kSmemBytes) kb = (kb + 1) / 2;
    const int k1 = k0 + kb;
    const int e = group_panel<Ops>(W, ld, n, k0, kb, piv, sm, pr, red_k, red_i, grp);
    if (info == 0) info = e;
    if (k1 >= n) break;
    // ---- U12 = L11^-1 A12 (rows [k0, k1), columns [k1, n)), a thread per column, 16 rows at a time in registers
    for (int e = tid; e < kb * kb; e += kBT) {
      const int r = e / kb, c = e % kb;
      L11[r * kMaxNB + c] = W[int64_t(k0 + r) * ld + k0 + c];
    }
    __syncthreads();
    for (int c = k1 + grp.thread(); c < n; c += grp.threads()) {
      T* col = W + int64_t(k0) * ld + c;
      for (int rb = 0; rb < kb; rb += 16) {
        T x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) x[r] = rb + r < kb ? col[int64_t(rb + r) * ld] : Ops::from_d(0.0);
        for (int t = 0; t < rb; ++t) {
          const T xt = col[int64_t(t) * ld];
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (rb + r < kb) Ops::fms(x[r], L11[(rb + r) * kMaxNB + t], xt);
        }
#pragma unroll
        for (int r = 1; r < 16; ++r)
          if (rb + r < kb)
#pragma unroll
            for (int t = 0; t < r; ++t) Ops::fms(x[r], L11[(rb + r) * kMaxNB + rb + t], x[t]);
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (rb + r < kb) col[int64_t(rb + r) * ld] = x[r];
      }
    }
    grp.sync();
    // ---- A22 -= L21 U12 in 64 x 64 tiles, 4 x 4 entries per thread; half a CTA takes a run of consecutive tiles, so that
    // it stages the rows of L21 seldom
    const int tr = ttid >> 4, tc = ttid & 15;
    const int tiles_c = (n - k1 + kTN - 1) / kTN, tiles = (n - k1 + kTM - 1) / kTM * tiles_c;
    const int who = grp.rank * kTeams + team, all = grp.ctas * kTeams;
    const int t0 = int(int64_t(tiles) * who / all), t1 = int(int64_t(tiles) * (who + 1) / all);
    int staged = -1;
    for (int t = t0; t < t1; ++t) {
      const int r0 = k1 + t / tiles_c * kTM, c0 = k1 + t % tiles_c * kTN;
      const int rows_t = min(kTM, n - r0), cols = min(kTN, n - c0);
      // thread (tr, tc) owns rows 4 tr .. 4 tr + 3 and four columns
      T acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int r = 4 * tr + a, c = Ops::column(tc, b);
          acc[a][b] = (r < rows_t && c < cols) ? W[int64_t(r0 + r) * ld + c0 + c] : Ops::from_d(0.0);
        }
      team_sync();  // the previous tile is done with L and U
      if (staged != r0) {
        for (int e = ttid; e < kTM * kb; e += kBT / kTeams) {
          const int r = e / kb, c = e % kb;
          if (r < rows_t) Ops::stage_l(tiles_s, r, c, W[int64_t(r0 + r) * ld + k0 + c]);
        }
        staged = r0;
      }
      for (int e = ttid; e < kb * kTN; e += kBT / kTeams) {
        const int r = e / kTN, c = e % kTN;
        if (c < cols) Ops::stage_u(tiles_s, r, c, W[int64_t(k0 + r) * ld + c0 + c]);
      }
      team_sync();
      Ops::tile_update(acc, tiles_s, 4 * tr, tc, kb);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int r = 4 * tr + a, c = Ops::column(tc, b);
          if (r < rows_t && c < cols) W[int64_t(r0 + r) * ld + c0 + c] = acc[a][b];
        }
    }
    grp.sync();  // the next panel reads what other CTAs updated, and writes over the staged tiles
  }
  return info;
}

// ---- triangular solves on a shared-memory vector ------------------------------------------------------------

// The row permutation of the interchanges: perm[i] is the row that ends up at i.  One thread, on shared memory (scratch:
// 2 n ints).
__device__ void permutation(const int32_t* piv, int n, int32_t* perm, int* scratch) {
  int *sp = scratch, *row = scratch + n;
  for (int i = threadIdx.x; i < n; i += kBT) {
    sp[i] = piv[i];
    row[i] = i;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int j = 0; j < n; ++j) {
      const int p = sp[j];
      if (p != j) { const int t = row[j]; row[j] = row[p]; row[p] = t; }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kBT) perm[i] = row[i];
  __syncthreads();
}

// v = U^-1 L^-1 v (v already permuted) with the factors in W.  The forward and backward substitutions go by blocks of 32
// rows: warp 0 solves a block's diagonal part (staged in shared memory), then all warps subtract the block's columns
// from the rows still to come (one warp per row, lanes over the block's columns, coalesced, four rows at a time).  In a
// cluster every CTA holds v, block b is solved and its rows are kept up to date by CTA b % ctas, and each solved block
// goes to all of them.
template <class Ops, bool COOP>
__device__ void group_lu_solve(const typename Ops::T* W, int64_t ld, int n, double* v, typename Ops::T (*diag)[33],
                               const Group<COOP>& grp) {
  using T = typename Ops::T;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + 31) / 32;
  auto stage = [&](int b0, int bs) {
    for (int e = tid; e < 32 * 32; e += kBT) {
      const int r = e >> 5, c = e & 31;
      if (r < bs && c < bs) diag[r][c] = W[int64_t(b0 + r) * ld + b0 + c];
    }
    __syncthreads();
  };
  auto publish = [&](int b0, int bs, double xv) {
    if (lane < bs) {
      v[b0 + lane] = xv;
      if constexpr (COOP)
        for (int c = 0; c < grp.ctas; ++c)
          if (c != grp.rank) Group<COOP>::put(Group<COOP>::remote(&v[b0 + lane], c), xv);
    }
  };
  // Rows of the blocks [q0, q1) that this CTA keeps: v[i] -= sum over the block at b0 of W[i][b0 + .] v[b0 + .], 16 rows a
  // warp.  The sums run over the lanes in halves (16, 8, 4, 2, 1 apart); each exchange also halves the rows that a lane
  // goes on with, which leaves the same additions in the same order but a third of the FP64 instructions.
  auto subtract = [&](int q0, int q1, int b0, int bs) {
    const double xb = lane < bs ? v[b0 + lane] : 0.0;
    const int first = COOP ? q0 + ((grp.rank - q0) % grp.ctas + grp.ctas) % grp.ctas : q0;
    const int step = COOP ? grp.ctas : 1;
    const int halves = first < q1 ? (q1 - first + step - 1) / step * 2 : 0;
    for (int k = warp; k < halves; k += kWarps) {
      const int i0 = (first + (k >> 1) * step) * 32 + (k & 1) * 16;
      double s[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        s[u] = (i0 + u < n && lane < bs) ? Ops::to_d(W[int64_t(i0 + u) * ld + b0 + lane]) * xb : 0.0;
#pragma unroll
      for (int h = 8; h > 0; h >>= 1) {  // lanes 2 h apart exchange; the upper one keeps the rows from h on
        const bool up = lane & (2 * h);
#pragma unroll
        for (int u = 0; u < h; ++u) {
          const double mine = up ? s[u + h] : s[u], theirs = up ? s[u] : s[u + h];
          s[u] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2 * h);
        }
      }
      const double total = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
      const int row = i0 + (lane >> 1);
      if ((lane & 1) == 0 && row < n) v[row] -= total;
    }
  };
  // forward: unit lower
  for (int q = 0; q < nblk; ++q) {
    const int b0 = q * 32, bs = min(32, n - b0);
    if (!COOP || grp.rank == q % grp.ctas) {
      stage(b0, bs);  // (its barrier also completes this CTA's updates of the block's rows)
      if (warp == 0) {
        double xv = lane < bs ? v[b0 + lane] : 0.0;
        for (int r = 1; r < bs; ++r) {
          const double lr = lane < r ? Ops::to_d(diag[r][lane]) : 0.0;
          double s = lr * xv;
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == r) xv -= s;
        }
        publish(b0, bs, xv);
      }
    }
    grp.sync();
    subtract(q + 1, nblk, b0, bs);
  }
  grp.sync();
  // backward: upper with its diagonal
  for (int q = nblk - 1; q >= 0; --q) {
    const int b0 = q * 32, bs = min(32, n - b0);
    if (!COOP || grp.rank == q % grp.ctas) {
      stage(b0, bs);
      if (warp == 0) {
        double xv = lane < bs ? v[b0 + lane] : 0.0;
        for (int r = bs - 1; r >= 0; --r) {
          const double ur = (lane > r && lane < bs) ? Ops::to_d(diag[r][lane]) : 0.0;
          double s = ur * xv;
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == r) xv = (xv - s) / Ops::to_d(diag[r][r]);
        }
        publish(b0, bs, xv);
      }
    }
    grp.sync();
    subtract(0, q, b0, bs);
  }
  grp.sync();
}

// r = b - K y (FP64, K the equilibrated matrix), returns max_i |r_i| / max_i (|K| |y| + |b|)_i.
template <bool COOP>
__device__ double group_residual(const double* K, int64_t ld, int n, const double* y, const double* b, double* r,
                                 double* red_v, Group<COOP>& grp) {
  const int lane = threadIdx.x & 31;
  double rmax = 0.0, smax = 0.0;
  for (int i = grp.warp(); i < n; i += grp.warps()) {
    const double* Ki = K + int64_t(i) * ld;
    double s = 0.0, a = 0.0;
    for (int c = lane; c < n; c += 32) {
      const double kv = Ki[c];
      s = fma(kv, y[c], s);
      a = fma(fabs(kv), fabs(y[c]), a);
    }
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      a += __shfl_xor_sync(0xffffffffu, a, o);
    }
    if (lane == 0) {
      const double ri = b[i] - s;
      r[i] = ri;
      rmax = fmax(rmax, fabs(ri));
      smax = fmax(smax, a + fabs(b[i]));
    }
  }
  rmax = cta_max(rmax, red_v);
  smax = cta_max(smax, red_v);
  int unused = 0;
  grp.argmax(rmax, unused);  // (its barrier also completes r for the other CTAs)
  grp.argmax(smax, unused);
  return smax > 0.0 ? rmax / smax : rmax;
}

// ---- one system -------------------------------------------------------------------------------------------------

template <class Ops, bool COOP>
__device__ void solve_system(const BatchSys& sys, char* slice, SmemLU& sm, PanelRows& pr, double* red_v, int* red_i,
                             BatchOut* out, Group<COOP>& grp) {
  using T = typename Ops::T;
  const int n = sys.n;
  const int64_t ld = (int64_t(n) + 3) & ~int64_t(3);
  double* K = reinterpret_cast<double*>(slice);
  T* W = reinterpret_cast<T*>(K + int64_t(n) * ld);
  double* A = reinterpret_cast<double*>(W + int64_t(n) * ld);
  double* dr = A + int64_t(n) * ld;
  double* dc = dr + n;
  double* b = dc + n;
  double* rv = b + n;
  int32_t* piv = reinterpret_cast<int32_t*>(rv + n);
  int32_t* perm = piv + n;
  double* part = reinterpret_cast<double*>(W);  // column maxima by CTA, before W is written
  switch (sys.p.rbf) {
    case UPDES_RBF_POLYHARMONIC: assemble_system<UPDES_RBF_POLYHARMONIC>(sys, K, A, ld, dr, dc, b, part, grp); break;
    case UPDES_RBF_GAUSSIAN: assemble_system<UPDES_RBF_GAUSSIAN>(sys, K, A, ld, dr, dc, b, part, grp); break;
    case UPDES_RBF_MULTIQUADRIC: assemble_system<UPDES_RBF_MULTIQUADRIC>(sys, K, A, ld, dr, dc, b, part, grp); break;
    case UPDES_RBF_INVERSE_MULTIQUADRIC:
      assemble_system<UPDES_RBF_INVERSE_MULTIQUADRIC>(sys, K, A, ld, dr, dc, b, part, grp); break;
    default: assemble_system<UPDES_RBF_THIN_PLATE>(sys, K, A, ld, dr, dc, b, part, grp); break;
  }
  scale_columns_to_w<Ops>(sys, K, W, ld, dc, grp);
  const int info = group_lu<Ops>(W, ld, n, COOP ? max(sys.nb, kCoopNB) : sys.nb, piv, sm, pr, reinterpret_cast<Key*>(red_v), red_i, grp);
  // shared memory from here on: y and the correction, a staged diagonal block
  double* y = reinterpret_cast<double*>(&sm);
  double* d = y + kMaxBatchN;
  T(*diag)[33] = reinterpret_cast<T(*)[33]>(d + kMaxBatchN);
  if (grp.rank == 0) permutation(piv, n, perm, reinterpret_cast<int*>(&sm));
  grp.sync();
  for (int i = threadIdx.x; i < n; i += kBT) y[i] = b[perm[i]];
  grp.sync();
  group_lu_solve<Ops>(W, ld, n, y, diag, grp);
  int sweeps = 0;
  double bwd = group_residual(K, ld, n, y, b, rv, red_v, grp);
  double last = INFINITY;
  while (bwd > kBwdStop && sweeps < sys.max_sweeps && bwd < 0.5 * last) {
    for (int i = threadIdx.x; i < n; i += kBT) d[i] = rv[perm[i]];
    grp.sync();
    group_lu_solve<Ops>(W, ld, n, d, diag, grp);
    for (int i = threadIdx.x; i < n; i += kBT) y[i] += d[i];
    __syncthreads();
    last = bwd;
    bwd = group_residual(K, ld, n, y, b, rv, red_v, grp);
    ++sweeps;
  }
  // coeffs = Dc y; vals = A[:N] coeffs
  for (int i = threadIdx.x; i < n; i += kBT) {
    const double c = dc[i] * y[i];
    if (grp.rank == 0) sys.coeffs[i] = c;
    y[i] = c;
  }
  __syncthreads();
  if (sys.vals) {
    const int lane = threadIdx.x & 31;
    for (int i = grp.warp(); i < sys.p.N; i += grp.warps()) {
      const double* Ai = A + int64_t(i) * ld;
      double s = 0.0;
      for (int c = lane; c < n; c += 32) s = fma(Ai[c], y[c], s);
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) sys.vals[i] = s;
    }
  }
  if (grp.thread() == 0) {
    out->lu_info = info;
    out->sweeps = sweeps;
    out->backward_error = bwd;
    out->converged = (info == 0 && bwd <= kBwdFloorB) ? 1 : 0;
    out->done = 1;
  }
  grp.sync();
}

// COOP: each cluster takes systems from the queue and solves them together, in the slice of its own; else each CTA.
template <bool COOP>
__global__ void __launch_bounds__(kBT) batched_solve_kernel(const BatchSys* __restrict__ systems,
                                                            const int32_t* __restrict__ order, int count,
                                                            int* __restrict__ queue, char* __restrict__ scratch,
                                                            size_t slice_bytes, BatchOut* __restrict__ outs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemLU& sm = *reinterpret_cast<SmemLU*>(smem_raw);
  __shared__ double red_v[kWarps];
  __shared__ int red_i[kWarps];
  __shared__ int s_next;
  __shared__ Exchange ex;
  __shared__ PanelRows pr;
  Group<COOP> grp;
  int team = blockIdx.x;
  if constexpr (COOP) {
    uint32_t rank, ctas;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
    grp.rank = int(rank);
    grp.ctas = int(ctas);
    grp.ex = &ex;
    team = blockIdx.x / int(ctas);
  }
  char* slice = scratch + size_t(team) * slice_bytes;
  for (;;) {
    if (grp.rank == 0 && threadIdx.x == 0) {
      const int k = atomicAdd(queue, 1);
      s_next = k;
      if constexpr (COOP)
        for (int c = 1; c < grp.ctas; ++c)
          asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(Group<COOP>::remote(&s_next, c)), "r"(k) : "memory");
    }
    grp.sync();
    const int k = s_next;
    grp.sync();
    if (k >= count) break;
    const int i = order[k];
    const BatchSys sys = systems[i];
    if (sys.precision == UPDES_PREC_FP64) solve_system<OpsF64>(sys, slice, sm, pr, red_v, red_i, outs + i, grp);
    else solve_system<OpsDF>(sys, slice, sm, pr, red_v, red_i, outs + i, grp);
  }
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// Bytes of one CTA's (cluster's) slice for systems of at most n_max unknowns: K, W and A (n x ld, 8 bytes each),
// four n-vectors, the pivots and the permutation.
size_t slice_bytes_for(int n_max) {
  const size_t ld = (size_t(n_max) + 3) & ~size_t(3);
  return align256(3 * size_t(n_max) * ld * 8 + 4 * size_t(n_max) * 8 + 2 * size_t(n_max) * 4);
}

int batch_n_max(const updes_problem* problems, int32_t count, int* n_max) {
  int mx = 0;
  for (int32_t i = 0; i < count; ++i) {
    const int e = updes_check_problem(&problems[i]);
    if (e) return e;
    if (problems[i].supports) return UPDES_ERR_UNSUPPORTED;
    mx = std::max(mx, problems[i].N + problems[i].M);
  }
  if (mx > kMaxBatchN) return UPDES_ERR_UNSUPPORTED;
  *n_max = mx;
  return UPDES_OK;
}

int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return sms;
}

std::atomic<unsigned long long> g_batched_smem_done[2];

// Who solves what, from the sizes alone: the systems of at least some size by clusters, the others by one CTA each on the SMs
// that no cluster holds and then on those that are done, with the size that gives the shortest launch by the times below.
// A cluster shortens one system (n = 2,031 from 353 to 49 ms, n = 790 from 30 to 8.6) but its eight SMs do less together,
// so it pays where a launch would wait for a few large systems and not where the SMs are full: 256 clouds of up to
// 2,025 nodes 376 ms with one CTA a system, 118 with clusters for the large ones; 152 systems of 784 nodes 30 ms with
// one CTA each, 84 on clusters (a rule by the average SM's share of n^3 took those: 127 of them 77 ms instead of 45). Below 384
// unknowns a cluster gains nothing.  With a CTA count given by the caller every system takes one CTA.
constexpr int kCoopMinN = 384;

// Milliseconds of a system on one CTA (batches of 64 and one at a time) and on a cluster, FP32; FP64 takes up to 2.3 times as
// long on either.
constexpr struct { double n, single, cluster; } kSystemMs[] = {
    {64, 0.55, 1.2}, {100, 0.9, 1.5}, {200, 2.1, 2.1}, {400, 7.0, 3.45}, {787, 29.5, 8.5},
    {1603, 172, 29.8}, {2028, 350, 48.9}, {3028, 1180, 125}, {4096, 3300, 280}};

double system_ms(int n, bool cluster) {
  const int last = int(sizeof kSystemMs / sizeof kSystemMs[0]) - 1;
  int i = 1;
  while (i < last && n > kSystemMs[i].n) ++i;
  const auto &a = kSystemMs[i - 1], &b = kSystemMs[i];
  const double x = (std::log(std::max(n, 1)) - std::log(a.n)) / (std::log(b.n) - std::log(a.n));
  const double ya = cluster ? a.cluster : a.single, yb = cluster ? b.cluster : b.single;
  return std::exp(std::log(ya) + x * (std::log(yb) - std::log(ya)));
}

// The launch of systems of sizes n (falling), those up to index `coop` on clusters: each goes to the first that is free.
double launch_ms(const std::vector<int>& n, size_t coop, int sms, int teams) {
  std::priority_queue<double, std::vector<double>, std::greater<double>> team, sm;
  const int held = int(std::min<size_t>(coop, size_t(teams)));
  for (int i = 0; i < held; ++i) team.push(0.0);
  double end = 0.0;
  for (size_t i = 0; i < coop; ++i) {
    const double t = team.top() + system_ms(n[i], true);
    team.pop();
    team.push(t);
    end = std::max(end, t);
  }
  for (int i = 0; i < sms - held * kMaxC; ++i) sm.push(0.0);
  for (; !team.empty(); team.pop())
    for (int i = 0; i < kMaxC; ++i) sm.push(team.top());
  for (size_t i = coop; i < n.size(); ++i) {
    const double t = sm.top() + system_ms(n[i], false);
    sm.pop();
    sm.push(t);
    end = std::max(end, t);
  }
  return end;
}

// The size from which systems go to clusters (INT_MAX: none) and the launch's time.  At most 24 sizes are tried.
int cluster_from(std::vector<int> n, int sms, int teams, double* ms) {
  std::sort(n.begin(), n.end(), std::greater<int>());
  *ms = launch_ms(n, 0, sms, 0);
  int from = INT_MAX;
  if (teams <= 0 || sms < teams * kMaxC) return from;
  std::vector<size_t> ends;  // behind the last system of each size
  for (size_t i = 0; i < n.size() && n[i] >= kCoopMinN; ++i)
    if (i + 1 == n.size() || n[i + 1] != n[i]) ends.push_back(i + 1);
  const size_t step = (ends.size() + 23) / 24;
  for (size_t k = 0; k < ends.size(); k += step) {
    const double t = launch_ms(n, ends[k], sms, teams);
    if (t < 0.98 * *ms) {
      *ms = t;
      from = n[ends[k] - 1];
    }
  }
  return from;
}

struct Split {
  int n_coop = 0, n_single = 0;      // largest size of either kind
  int coop = 0, single = 0;          // systems
  int teams = 0, ctas = 0;           // clusters; CTAs for the others
  int from = INT_MAX;                // size from which a system is solved by a cluster
  bool by_cluster(int n) const { return n >= from; }
  size_t coop_slice() const { return coop ? slice_bytes_for(n_coop) : 0; }
  size_t single_slice() const { return single ? slice_bytes_for(n_single) : 0; }
  size_t slices() const { return coop_slice() * size_t(teams) + single_slice() * size_t(ctas); }
};

// Clusters of kMaxC CTAs that fit the device at once (0: none).
int max_teams() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (const int v = known[dev].load()) return v - 1;
  const void* kern = (const void*)batched_solve_kernel<true>;
  int n = 0;
  if (smem_opt_in(kern, int(kSmemBytes), g_batched_smem_done[1]) == UPDES_OK) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {unsigned(kMaxC), 1, 1};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kMaxC);
    cfg.blockDim = dim3(kBT);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) n = 0;
    (void)cudaGetLastError();
  }
  known[dev].store(n + 1);
  return n;
}

Split split_batch(const updes_problem* problems, int32_t count, int32_t ctas) {
  Split s;
  const int sms = sm_count(), teams = ctas > 0 ? 0 : max_teams();
  if (teams > 0) {
    std::vector<int> n(count);
    for (int32_t i = 0; i < count; ++i) n[i] = problems[i].N + problems[i].M;
    double ms;
    s.from = cluster_from(std::move(n), sms, teams, &ms);
  }
  for (int32_t i = 0; i < count; ++i) {
    const int n = problems[i].N + problems[i].M;
    if (s.by_cluster(n)) {
      ++s.coop;
      s.n_coop = std::max(s.n_coop, n);
    } else {
      ++s.single;
      s.n_single = std::max(s.n_single, n);
    }
  }
  s.teams = std::min(teams, s.coop);
  s.ctas = std::min(ctas > 0 ? int(ctas) : sms, s.single);
  return s;
}

}  // namespace

namespace {
size_t tables_bytes_for(int32_t count) {
  return align256(size_t(count) * (sizeof(BatchSys) + sizeof(BatchOut) + 4)) + 1024;
}
}  // namespace

extern "C" int updes_solve_batched_plan(const int32_t* n, int32_t count, int32_t sms, int32_t teams, int32_t* from,
                                        double* ms) {
  if (!n || count <= 0 || sms < 0 || teams < 0 || !from || !ms) return UPDES_ERR_INVALID;
  for (int32_t i = 0; i < count; ++i)
    if (n[i] <= 0 || n[i] > kMaxBatchN) return UPDES_ERR_UNSUPPORTED;
  if (sms == 0) {
    sms = sm_count();
    teams = max_teams();
    if (sms <= 0) return UPDES_ERR_CUDA;
  }
  *from = cluster_from(std::vector<int>(n, n + count), sms, teams, ms);
  return UPDES_OK;
}

extern "C" int updes_solve_batched_tables(int32_t count, size_t* bytes) {
  if (count <= 0 || !bytes) return UPDES_ERR_INVALID;
  *bytes = tables_bytes_for(count);
  return UPDES_OK;
}

extern "C" int updes_solve_batched_workspace(const updes_problem* problems, int32_t count, int32_t ctas,
                                             size_t* bytes) {
  if (!problems || count <= 0 || ctas < 0 || !bytes) return UPDES_ERR_INVALID;
  int n_max = 0;
  const int e = batch_n_max(problems, count, &n_max);
  if (e) return e;
  if (sm_count() <= 0) return UPDES_ERR_CUDA;
  *bytes = split_batch(problems, count, ctas).slices() + 256 + tables_bytes_for(count);
  return UPDES_OK;
}

namespace {
struct PendingBatch {
  std::vector<BatchSys> sys;  // copied from by the stream
  std::vector<int32_t> order;
  const BatchOut* d_out;
};
}  // namespace

extern "C" int updes_solve_batched_begin(const updes_problem* problems, int32_t count, const double* const* q,
                                         double* const* coeffs, double* const* vals, const int32_t* precision,
                                         const int32_t* panel_width, int32_t max_sweeps, int32_t ctas, void* workspace,
                                         size_t workspace_bytes, void* tables, size_t tables_bytes, void* stream,
                                         void** pending) {
  if (!pending) return UPDES_ERR_INVALID;
  *pending = nullptr;
  if (!tables || count <= 0) return UPDES_ERR_INVALID;
  if (tables_bytes < tables_bytes_for(count)) return UPDES_ERR_WORKSPACE;
  if (!problems || count <= 0 || !q || !coeffs || !workspace || ctas < 0 || max_sweeps < 0) return UPDES_ERR_INVALID;
  int n_max = 0;
  int e = batch_n_max(problems, count, &n_max);
  if (e) return e;
  if (sm_count() <= 0) return UPDES_ERR_CUDA;
  const Split split = split_batch(problems, count, ctas);
  if (workspace_bytes < split.slices() + 256) return UPDES_ERR_WORKSPACE;
  std::unique_ptr<PendingBatch> h(new (std::nothrow) PendingBatch);
  if (!h) return UPDES_ERR_CUDA;
  h->sys.resize(count);
  h->order.resize(count);
  std::vector<BatchSys>& sys = h->sys;
  for (int32_t i = 0; i < count; ++i) {
    if (!q[i] || !coeffs[i]) return UPDES_ERR_INVALID;
    const int pr = precision ? precision[i] : UPDES_PREC_FP32;
    const int nb = panel_width ? panel_width[i] : 16;
    if ((pr != UPDES_PREC_FP32 && pr != UPDES_PREC_FP64) || nb < 1 || nb > kMaxNB) return UPDES_ERR_INVALID;
    sys[i].p = problems[i];
    sys[i].q = q[i];
    sys[i].coeffs = coeffs[i];
    sys[i].vals = vals ? vals[i] : nullptr;
    sys[i].n = problems[i].N + problems[i].M;
    sys[i].nb = nb;
    sys[i].precision = pr;
    sys[i].max_sweeps = max_sweeps;
  }
  // the clusters' systems, then the others, each largest first (their solves are the longest)
  std::vector<int32_t>& order = h->order;
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
    const bool ta = split.by_cluster(sys[a].n), tb = split.by_cluster(sys[b].n);
    if (ta != tb) return ta;
    const double ca = double(sys[a].n) * sys[a].n * sys[a].n * (sys[a].precision == UPDES_PREC_FP64 ? 6.0 : 1.0);
    const double cb = double(sys[b].n) * sys[b].n * sys[b].n * (sys[b].precision == UPDES_PREC_FP64 ? 6.0 : 1.0);
    return ca > cb;
  });
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  char* meta = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(tables) + 255) & ~uintptr_t(255));
  BatchSys* d_sys = reinterpret_cast<BatchSys*>(meta);
  BatchOut* d_out = reinterpret_cast<BatchOut*>(meta + align256(size_t(count) * sizeof(BatchSys)));
  int32_t* d_order = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(d_out) + align256(size_t(count) * sizeof(BatchOut)));
  int* d_queue = d_order + count;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  UPDES_CUDA_TRY(cudaMemcpyAsync(d_sys, sys.data(), sizeof(BatchSys) * count, cudaMemcpyHostToDevice, s));
  UPDES_CUDA_TRY(cudaMemcpyAsync(d_order, order.data(), sizeof(int32_t) * count, cudaMemcpyHostToDevice, s));
  UPDES_CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(BatchOut) * count, s));
  UPDES_CUDA_TRY(cudaMemsetAsync(d_queue, 0, 2 * sizeof(int), s));
  if ((e = smem_opt_in((const void*)batched_solve_kernel<false>, int(kSmemBytes), g_batched_smem_done[0]))) return e;
  {
    double flops = 0.0;
    for (const auto& x : sys) flops += 2.0 / 3.0 * double(x.n) * x.n * x.n;
    StatScope sc(kStatOther, s, flops, 0.0);
    SideStream side;
    const bool both = split.teams > 0 && split.ctas > 0;
    if (both && ((e = side.create(s)) || (e = side.start()))) return e;
    if (split.teams > 0) {
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim = {unsigned(kMaxC), 1, 1};
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(unsigned(split.teams * kMaxC));
      cfg.blockDim = dim3(kBT);
      cfg.dynamicSmemBytes = kSmemBytes;
      cfg.stream = both ? side.side : s;  // of higher priority: the clusters start first
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      UPDES_CUDA_TRY(cudaLaunchKernelEx(&cfg, batched_solve_kernel<true>, (const BatchSys*)d_sys, (const int32_t*)d_order,
                                        split.coop, d_queue, base, split.coop_slice(), d_out));
      stats_count_launch(1);
    }
    if (split.ctas > 0) {
      batched_solve_kernel<false><<<split.ctas, kBT, kSmemBytes, s>>>(
          d_sys, d_order + split.coop, split.single, d_queue + 1, base + split.coop_slice() * size_t(split.teams),
          split.single_slice(), d_out);
      UPDES_LAUNCH_CHECK();
    }
    if (both && (e = side.finish())) return e;
  }
  h->d_out = d_out;
  *pending = h.release();
  return UPDES_OK;
}

extern "C" int updes_solve_batched_end(void* pending, updes_solve_info* infos, void* stream) {
  if (!pending) return UPDES_ERR_INVALID;
  std::unique_ptr<PendingBatch> h(static_cast<PendingBatch*>(pending));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int32_t count = int32_t(h->sys.size());
  std::vector<BatchOut> outs(count);
  UPDES_CUDA_TRY(cudaMemcpyAsync(outs.data(), h->d_out, sizeof(BatchOut) * count, cudaMemcpyDeviceToHost, s));
  UPDES_CUDA_TRY(cudaStreamSynchronize(s));
  int status = UPDES_OK;
  for (int32_t i = 0; i < count; ++i) {
    if (infos) {
      std::memset(&infos[i], 0, sizeof(updes_solve_info));
      infos[i].iters = outs[i].sweeps;
      infos[i].lu_info = outs[i].lu_info;
      infos[i].converged = outs[i].converged;
      infos[i].backward_error = outs[i].backward_error;
    }
    if (!outs[i].done) status = UPDES_ERR_CUDA;
    else if (status == UPDES_OK && outs[i].lu_info) status = UPDES_ERR_SINGULAR;
  }
  return status;
}

extern "C" int updes_solve_batched(const updes_problem* problems, int32_t count, const double* const* q,
                                   double* const* coeffs, double* const* vals, const int32_t* precision,
                                   const int32_t* panel_width, int32_t max_sweeps, int32_t ctas,
                                   updes_solve_info* infos, void* workspace, size_t workspace_bytes, void* stream) {
  if (!problems || count <= 0 || !workspace || ctas < 0) return UPDES_ERR_INVALID;
  size_t need = 0;
  if (int e = updes_solve_batched_workspace(problems, count, ctas, &need)) return e;
  if (workspace_bytes < need) return UPDES_ERR_WORKSPACE;
  // the tables behind the systems' slices
  const size_t tb = tables_bytes_for(count);
  void* pending = nullptr;
  const int e = updes_solve_batched_begin(problems, count, q, coeffs, vals, precision, panel_width, max_sweeps, ctas,
                                          workspace, need - tb, static_cast<char*>(workspace) + (need - tb), tb, stream, &pending);
  return e ? e : updes_solve_batched_end(pending, infos, stream);
}
