// Tensor-core trailing update of the FP64 LU (sm_103a):
//
//   C  <-  C - A * B        C, A (m x K, a block of L), B (K x nc, a block of U): FP64, K <= 256
//
// Why.  GB300's FP64 pipe does two multiply-adds a cycle and SM, so an FP64 GEMM on it (64 x 64 SIMT tiles, 97 % of
// that rate) took 552 of the 690 ms of an N = 10,000 solve.  The bf16 tensor cores do 4,096, exactly, on small
// integers.
//
// Numerics.  Every operand is written as 7 bf16 integer digits under a power-of-two scale shared by a row of A (a
// column of B) over all of K:
//   a = 2^(e - 55) * sum_i d_i 2^(8 (6 - i)),   |d_i| <= 128,   |a| < 2^e for the whole row,
// by rounding the 53-bit significand to a multiple of 2^(e - 55): exact for entries within a factor 8 of the row's
// largest, cut at 2^-56 of 2^e otherwise (an FP64 rounding of that largest entry is 2^-54).  The cut is harmless where the
// entries that meet in a sum are of one size, as in K scaled by solve.cu (row_scale_kernel); where a row's largest entry
// meets small ones only (graded rows of a matrix that nobody scaled) it loses digits that a chain of FP64 multiply-adds
// keeps, so such matrices are factored with that (gemm64_chain_kernel in lu.cu).
// The digit products of equal weight 2^-8g, g = a + b <= 7 (34 of them), are summed in one FP32 accumulator over all of K:
// 256 products of at most 2^14 each, at most 7 times, so sums stay integers below 2^24.8 and are exact unless
// nearly every digit of a row and a column is at its limit with one sign, when the error is a unit of that group.
// Products with g >= 8 lie 2^-64 below 2^(ea + eb) each and are left out.  (The products with g = 7 are needed: the
// factors of an N = 600 r^3 system without them give coefficients with 3.5e-10 of error, a chain of FP64
// multiply-adds 1.1e-10, with them 1.2e-11.)  The eight sums make one 64-bit integer, which is converted and subtracted
// from C with one fused multiply-add: one rounding of the whole K-term sum and one of C, where a chain of FP64
// multiply-adds rounds K times.
// A row or column with a non-finite entry gets a NaN scale, so its part of C becomes NaN as in FP64 arithmetic.
//
// Structure.  A pre-pass writes the digits (A as [7][m][Kp], B transposed as [7][nc][Kp], Kp = K rounded up to 32)
// and the exponents.  The main kernel is persistent, one CTA an SM, tiles of 128 x 64 round robin:
//   warp 0     TMA producer: all digits of a 32-wide k block (7 x (8 + 4) KB = 84 KB, 64B swizzle) into a 2-stage
//              ring.  The whole stage is one box for A and one for B.
//   warp 1     MMA issuer: 12 instructions for the 34 products, x 2 k-steps, of tcgen05.mma (kind::f16, M = 128, N up to
//              256: several digit planes of B side by side) into 8 groups of 64 columns (all 512 TMEM columns: no second set);
//   warps 2-9  epilogue: read the 8 groups, make 64-bit integers of them and release the accumulators (the MMAs of the
//              next tile start then, their operands already in the ring); C, 32 columns at a time, through a
//              shared-memory transposition so that its rows are read and written whole.
// Bound by shared memory: a k-step reads 112 KB of operands there (as 34 MMAs of N = 64 it was 204 KB, 26,000 cycles a
// tile; all updates of an n = 10,006 factorisation then took 52 ms, now 45) and needs 1,088 cycles of MMAs; the epilogue needs two
// FP64-pipe operations an element (8,192 cycles a tile) beside them.
#include <algorithm>
#include <atomic>

#include "gemm_tc.cuh"
#include "stats.cuh"
#include "tc.cuh"

namespace {

constexpr int TM = 128, TN = 64, TK = 32;
constexpr int kDigits = 7, kGroups = 8;
constexpr int kStages = 2;
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr uint32_t kTmemCols = 512;
constexpr int kAPlane = TM * TK * 2, kBPlane = TN * TK * 2;          // 8 KB, 4 KB
constexpr int kStageBytes = kDigits * (kAPlane + kBPlane);           // 84 KB
constexpr int kCols = 32, kLdv = kCols + 1;                          // columns of a transposition pass
constexpr int kVBytes = TM * kLdv * 8;
constexpr int kSmemBytes = kStages * kStageBytes + kVBytes + 1024;
static_assert(kSmemBytes <= 226 * 1024, "shared memory");
constexpr int kNanExp = 1 << 20;  // exponent of a row or column with a non-finite entry

// instruction descriptor: D = F32, A = B = BF16, both K-major, M = 128
constexpr uint32_t idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(TM >> 4) << 24);
}

__device__ __forceinline__ void mma_acc(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(id), "r"(acc)
      : "memory");
}

// ---- digit pre-pass ------------------------------------------------------------------------------------
// Exponent field of |v| (1 for subnormals), 0x7ff for non-finite values, 0 for zero.
__device__ __forceinline__ int exp_field(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
  if (b == 0) return 0;
  return max(int(b >> 52), 1);
}

// Digits of v under the row's largest exponent field emax (1..0x7fe): v = 2^(emax - 1022 - 55) X + cut, X an
// integer below 2^55 in magnitude, written as balanced base-256 digits d[0] (leading) .. d[6].
__device__ __forceinline__ void digits_of(double v, int emax, int d[kDigits]) {
  const long long b = __double_as_longlong(v);
  const int e = exp_field(v);
  long long x = (b & 0xfffffffffffffll) | (int((b >> 52) & 0x7ff) ? 1ll << 52 : 0ll);
  const int sh = e - emax + 2;  // at most 2
  if (sh >= 0) x <<= sh;
  else if (sh > -56) x = (x + (1ll << (-sh - 1))) >> -sh;
  else x = 0;
  if (e == 0) x = 0;
  if (b < 0) x = -x;
#pragma unroll
  for (int i = kDigits - 1; i > 0; --i) {
    d[i] = int(static_cast<signed char>(x & 0xff));
    x = (x - d[i]) >> 8;
  }
  d[0] = int(x);
}

// Bits of the bf16 of an integer of at most 128 in magnitude (exact), in the low half: the integer added to
// 1.5 * 2^23 sits in the significand's low bits, the subtraction is exact.
__device__ __forceinline__ uint32_t bf16_bits(int d) {
  return __float_as_uint(__int_as_float(0x4b400000 + d) - 12582912.0f) >> 16;
}

// The exponent written for a row or column whose largest field is emax: its entries are below 2^e.
__device__ __forceinline__ int scale_exp(int emax) { return emax >= 0x7ff ? kNanExp : emax - 1022; }

// The digits of 8 consecutive entries under the exponent field emax, one 16-byte word into each of the 7 planes.
__device__ __forceinline__ void write_digits(const double* v, int emax, uint16_t* dst, int64_t plane) {
  uint32_t w[kDigits][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int d[kDigits];
    digits_of(emax >= 0x7ff ? 0.0 : v[i], max(emax, 1), d);
#pragma unroll
    for (int p = 0; p < kDigits; ++p) {
      const uint32_t h = bf16_bits(d[p]);
      if (i & 1) w[p][i >> 1] |= h << 16;
      else w[p][i >> 1] = h;
    }
  }
#pragma unroll
  for (int p = 0; p < kDigits; ++p)
    *reinterpret_cast<uint4*>(dst + p * plane) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// A (m x K, lda) -> Ad[p][r][k] and Ae[r]; 8 consecutive k a lane, `span` lanes (a power of two >= Kp / 8) a row.
__device__ __forceinline__ void digits_rows(int bx, const double* A, int64_t lda, int m, int K, int Kp,
                                            int span, uint16_t* __restrict__ Ad, int* __restrict__ Ae) {
  const int64_t t = int64_t(bx) * blockDim.x + threadIdx.x;
  const int r = int(t / span), q = int(t % span), k0 = q * 8;
  const bool ok = r < m;
  double v[8];
  int emax = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = (ok && k0 + i < K) ? A[int64_t(r) * lda + k0 + i] : 0.0;
    emax = max(emax, exp_field(v[i]));
  }
  for (int o = span >> 1; o > 0; o >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  if (!ok || k0 >= Kp) return;
  if (q == 0) Ae[r] = scale_exp(emax);
  write_digits(v, emax, Ad + int64_t(r) * Kp + k0, int64_t(m) * Kp);
}

// B (K x nc, ldb) -> Bd[p][c][k] and Be[c]; a lane a column, a warp 32 consecutive k, Kp / 32 warps a group of 32
// columns, 8 / (Kp / 32) groups a block.
__device__ __forceinline__ void digits_cols(int bx, const double* B, int64_t ldb, int nc, int K, int Kp,
                                            uint16_t* __restrict__ Bd, int* __restrict__ Be) {
  __shared__ int s_max[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = Kp / 32, groups = 8 / nw;
  const int grp = warp / nw, part = warp % nw;
  const int c = (bx * groups + grp) * 32 + lane, k0 = part * 32;
  const bool ok = grp < groups && c < nc;
  double v[32];
  int emax = 0;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    v[i] = (ok && k0 + i < K) ? B[int64_t(k0 + i) * ldb + c] : 0.0;
    emax = max(emax, exp_field(v[i]));
  }
  s_max[warp][lane] = emax;
  __syncthreads();
  if (!ok) return;
  for (int w = 0; w < nw; ++w) emax = max(emax, s_max[grp * nw + w][lane]);
  if (part == 0) Be[c] = scale_exp(emax);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    write_digits(v + j * 8, emax, Bd + int64_t(c) * Kp + k0 + j * 8, int64_t(nc) * Kp);
  }
}

// Both digit passes of an update in one launch: blocks [0, row_blocks) take rows of A, the others columns of B.
__global__ void __launch_bounds__(256) digits64_kernel(const double* A, int64_t lda, int m, const double* B, int64_t ldb, int nc, int K,
                                                       int Kp, int span, int row_blocks, uint16_t* __restrict__ Ad,
                                                       int* __restrict__ Ae, uint16_t* __restrict__ Bd,
                                                       int* __restrict__ Be) {
  allow_next();
  wait_previous();
  const int b = int(blockIdx.x);
  if (b < row_blocks) digits_rows(b, A, lda, m, K, Kp, span, Ad, Ae);
  else digits_cols(b - row_blocks, B, ldb, nc, K, Kp, Bd, Be);
}

// ---- main kernel ---------------------------------------------------------------------------------------
struct Ctrl {
  uint64_t full[kStages], empty[kStages], tfull, tempty;
  uint32_t tmem;
  int abort_flag;
};

// The same barrier with a vote, so that the epilogue's warps leave together.
__device__ __forceinline__ bool epilogue_any(bool v) {
  uint32_t any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 1, %2, q;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(any)
      : "r"(uint32_t(v)), "n"(kEpiWarps * 32)
      : "memory");
  return any != 0;
}
__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory"); }

// v as a double (one rounding), divided by 2^8 if `fine` (by its exponent: v is an integer)
__device__ __forceinline__ double to_double(long long v, uint32_t fine) {
  const long long b = __double_as_longlong(double(v));
  return __longlong_as_double(fine && v != 0 ? b - (8ll << 52) : b);
}

// c + sign d 2^(ea + eb - 54); the power as one factor where it is a normal number
template <int SIGN>
__device__ __forceinline__ double add_scaled(double c, double d, int ea, int eb) {
  const int e = ea + eb - 54;
  if (e > -1022 && e < 1023) {
    const double f = __longlong_as_double(static_cast<long long>(e + 1023) << 52);
    return fma(SIGN > 0 ? f : -f, d, c);
  }
  if (ea >= kNanExp || eb >= kNanExp) return __longlong_as_double(0x7ff8000000000000ll);
  return SIGN > 0 ? c + scalbn(d, e) : c - scalbn(d, e);
}

// The MMAs of one 32-wide k block; `later` is false for the first block of a sum, whose first product in each group
// overwrites the accumulator.  The digit planes of B lie behind one another and so do the groups: one instruction
// multiplies digit plane a by up to four planes b, b + 1, ... into groups a + b, a + b + 1, ..., 12 instructions for 34
// products that read A 12 times.
__device__ __forceinline__ void mma_stage(uint32_t tmem, const uint8_t* sA, bool later) {
  const uint64_t a0 = make_desc(smem_u32(sA)), b0 = make_desc(smem_u32(sA + kDigits * kAPlane));
#pragma unroll
  for (int a = 0; a < kDigits; ++a) {
    const int planes = kGroups - a < kDigits ? kGroups - a : kDigits;
#pragma unroll
    for (int b = 0; b < planes;) {
      // group 7 begins with a = 1, b = 6, where groups 5 and 6 have their second product: an instruction of its own
      const int to = b + 4 < planes ? b + 4 : (a == 1 && b == 4) ? kDigits - 1 : planes;
#pragma unroll
      for (int kk = 0; kk < TK / 16; ++kk) {  // a k-step is 32 bytes: 2 descriptor units
        const bool first = kk == 0 && (a == 0 || (a == 1 && b == kDigits - 1));
        mma_acc(tmem + uint32_t((a + b) * TN), a0 + uint64_t(a * (kAPlane >> 4) + kk * 2),
                b0 + uint64_t(b * (kBPlane >> 4) + kk * 2), idesc((to - b) * TN), first ? uint32_t(later) : 1u);
      }
      b = to;
    }
  }
}

// The thread's row of 32 sums as integers.  x is the sum in units of group 5 (at most 2^62), r what groups 6 and 7 add
// to it, in units of group 7.  Where x has fewer than 54 bits the integer is in units of group 6 instead, so that its
// conversion to a double is what rounds either way; the result's bit of that column is set then.
__device__ __forceinline__ uint32_t read_sums(uint32_t taddr, long long* v) {
  uint32_t fine = 0;
#pragma unroll
  for (int ch = 0; ch < kCols / 8; ++ch) {
    float g[kGroups][8];
#pragma unroll
    for (int gi = 0; gi < kGroups; ++gi) tmem_ld8(taddr + uint32_t(gi * TN + ch * 8), g[gi]);
    tmem_wait_ld();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      long long x = __float2int_rn(g[0][u]);
#pragma unroll
      for (int gi = 1; gi < kGroups - 2; ++gi) x = (x << 8) + __float2int_rn(g[gi][u]);
      const long long r = (static_cast<long long>(__float2int_rn(g[6][u])) << 8) + __float2int_rn(g[7][u]);
      const bool f = x < (1ll << 54) && x > -(1ll << 54);
      v[ch * 8 + u] = f ? (x << 8) + ((r + 128) >> 8) : x + ((r + (1 << 15)) >> 16);
      fine |= uint32_t(f) << (ch * 8 + u);
    }
  }
  return fine;
}

__global__ void __launch_bounds__(kThreads, 1)
    ozaki64_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const int* Ae, const int* Be, double* C, int64_t ldc, int m,
                   int nc, int Kp, DeviceStatus* st) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  double(*sV)[kLdv] = reinterpret_cast<double(*)[kLdv]>(smem + kStages * kStageBytes);
  __shared__ Ctrl ctl;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_n = int(ceil_div(nc, TN)), tiles_m = int(ceil_div(m, TM));
  const int ntiles = tiles_n * tiles_m;
  const int nkb = Kp / TK;
  volatile int* abort_flag = &ctl.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 1);
    }
    mbar_init(&ctl.tfull, 1);
    mbar_init(&ctl.tempty, kEpiWarps);
    ctl.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  allow_next();
  wait_previous();
  const uint32_t tmem = ctl.tmem;
  int committed = 0;  // MMA issuer: k blocks committed so far

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint64_t keep = l2_policy_evict_last();
      int j = 0;
      for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
        const int r0 = (t / tiles_n) * TM, c0 = (t % tiles_n) * TN;
        for (int kb = 0; kb < nkb; ++kb, ++j) {
          const int s = j % kStages;
          if (!mbar_wait(&ctl.empty[s], (uint32_t(j / kStages) & 1u) ^ 1u, abort_flag)) {
            if (!*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 51); }
            *abort_flag = 1;
            break;
          }
          uint8_t* sA = smem + s * kStageBytes;
          mbar_expect_tx(&ctl.full[s], uint32_t(kStageBytes));
          tma_load_3d(smem_u32(sA), &tmA, kb * TK, r0, 0, &ctl.full[s], keep);
          tma_load_3d(smem_u32(sA + kDigits * kAPlane), &tmB, kb * TK, c0, 0, &ctl.full[s], keep);
        }
      }
      if (*abort_flag) {
        // copies still in flight must land before the CTA's shared memory goes away (bounded)
        for (int jj = (j > kStages ? j - kStages : 0); jj < j; ++jj) {
          for (long long it = 0; it < (1 << 22); ++it) {
            if (mbar_try_wait(&ctl.full[jj % kStages], uint32_t(jj / kStages) & 1u)) break;
            __nanosleep(64);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int j = 0, tl = 0;
      for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x, ++tl) {
        for (int kb = 0; kb < nkb; ++kb, ++j) {
          const int s = j % kStages;
          if ((kb == 0 && !mbar_wait(&ctl.tempty, (uint32_t(tl) & 1u) ^ 1u, abort_flag)) ||
              !mbar_wait(&ctl.full[s], uint32_t(j / kStages) & 1u, abort_flag)) {
            if (!*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 52); }
            *abort_flag = 1;
            break;
          }
          tc_fence_after();
          mma_stage(tmem, smem + s * kStageBytes, kb > 0);
          mma_commit(&ctl.empty[s]);
          if (kb == nkb - 1) mma_commit(&ctl.tfull);
          committed = j + 1;
        }
      }
    }
  } else {
    // ---------------- epilogue: lane quarter q = warp % 4, column half h ----------------
    const int q = warp & 3, h = (warp - 2) >> 2, ew = warp - 2;
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    int tl = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++tl) {
      const int r0 = (t / tiles_n) * TM, c0 = (t % tiles_n) * TN;
      // every wait ends in a warp vote, so a warp always leaves together (tcgen05.ld needs all 32 lanes)
      if (!__all_sync(0xffffffffu, mbar_wait(&ctl.tfull, uint32_t(tl) & 1u, abort_flag))) {
        if (lane == 0 && !*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 53); }
        *abort_flag = 1;
      }
      tc_fence_after();
      long long v[kCols];
      const uint32_t fine = read_sums(tmem + lane_base + uint32_t(h * kCols), v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.tempty);
      // C, 32 columns at a time: the warps that hold them write their integers, then every warp takes 16 rows
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const int c = c0 + half * kCols + lane;
        const int eb = c < nc ? __ldcg(Be + c) : 0;
        const int er = r0 + ew * 16 + (lane & 15), ea = er < m ? __ldcg(Ae + er) : 0;  // row i's in lane i
        double* cp = C + int64_t(r0 + ew * 16) * ldc + c;
        double old[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          old[i] = (c < nc && r0 + ew * 16 + i < m) ? __ldcs(cp + int64_t(i) * ldc) : 0.0;
        if (h == half) {
#pragma unroll
          for (int u = 0; u < kCols; ++u) sV[q * 32 + lane][u] = to_double(v[u], (fine >> u) & 1u);
        }
        epilogue_barrier();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int r = r0 + ew * 16 + i, e = __shfl_sync(0xffffffffu, ea, i);
          if (c < nc && r < m && !*abort_flag)
            __stcs(cp + int64_t(i) * ldc, add_scaled<-1>(old[i], sV[ew * 16 + i][lane], e, eb));
        }
        if (half == 0) epilogue_barrier();
      }
      if (epilogue_any(*abort_flag != 0)) break;
    }
  }

  // ---- teardown: all roles done; make sure no MMA is in flight before tensor memory is freed ----
  __syncthreads();
  if (warp == 1) {
    if (ctl.abort_flag && lane == 0 && committed > 0) {
      // MMAs complete in order: once the last commit has arrived nothing reads tensor memory (bounded)
      const int jj = committed - 1;
      for (long long it = 0; it < (1 << 22); ++it) {
        if (mbar_try_wait(&ctl.empty[jj % kStages], uint32_t(jj / kStages) & 1u)) break;
        __nanosleep(64);
      }
    }
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- a fixed matrix times up to 64 columns ------------------------------------------------------------------
// Y = A X for an m x n matrix whose digits are written once (updes_batch_prepare) and X of at most 64 columns: the
// same products and sums as above over k blocks of 256, each block's sum rounded once and added in FP64.  A 64-column
// product reads 14 bytes of digits an entry of A and is bound by its operands' way through shared memory, about
// a tenth of what double-float multiply-adds on the FP32 pipes cost.  The k blocks are split over `splits` CTAs a row
// tile, their sums added in order by the caller.
constexpr int kBlockK = 256;

__global__ void __launch_bounds__(kThreads, 1)
    rhs64_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const int* __restrict__ Ae, const int* __restrict__ Be, double* __restrict__ partial, int m, int nkb,
                 int splits, DeviceStatus* st, const int32_t* __restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ Ctrl ctl;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int items = int(ceil_div(m, TM)) * splits;
  volatile int* abort_flag = &ctl.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 1);
    }
    mbar_init(&ctl.tfull, 1);
    mbar_init(&ctl.tempty, kEpiWarps);
    ctl.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl.tmem;
  int committed = 0;
  auto first_block = [&](int item) { return int(int64_t(nkb) * (item % splits) / splits); };
  auto end_block = [&](int item) { return int(int64_t(nkb) * (item % splits + 1) / splits); };

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t stream = l2_policy_evict_first(), keep = l2_policy_evict_last();
      int j = 0;
      for (int it = blockIdx.x; it < items && !*abort_flag; it += gridDim.x) {
        const int r0 = (it / splits) * TM;
        for (int ks = first_block(it) * (kBlockK / TK); ks < end_block(it) * (kBlockK / TK); ++ks, ++j) {
          const int s = j % kStages;
          if (!mbar_wait(&ctl.empty[s], (uint32_t(j / kStages) & 1u) ^ 1u, abort_flag)) {
            if (!*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 54); }
            *abort_flag = 1;
            break;
          }
          uint8_t* sA = smem + s * kStageBytes;
          mbar_expect_tx(&ctl.full[s], uint32_t(kStageBytes));
          tma_load_3d(smem_u32(sA), &tmA, ks * TK, r0, 0, &ctl.full[s], stream);
          tma_load_3d(smem_u32(sA + kDigits * kAPlane), &tmB, ks * TK, 0, 0, &ctl.full[s], keep);
        }
      }
      if (*abort_flag) {
        // copies still in flight must land before the CTA's shared memory goes away (bounded)
        for (int jj = (j > kStages ? j - kStages : 0); jj < j; ++jj) {
          for (long long k = 0; k < (1 << 22); ++k) {
            if (mbar_try_wait(&ctl.full[jj % kStages], uint32_t(jj / kStages) & 1u)) break;
            __nanosleep(64);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int j = 0, sums = 0;
      for (int it = blockIdx.x; it < items && !*abort_flag; it += gridDim.x) {
        for (int kb = first_block(it); kb < end_block(it) && !*abort_flag; ++kb, ++sums) {
          for (int i = 0; i < kBlockK / TK; ++i, ++j) {
            const int s = j % kStages;
            if ((i == 0 && !mbar_wait(&ctl.tempty, (uint32_t(sums) & 1u) ^ 1u, abort_flag)) ||
                !mbar_wait(&ctl.full[s], uint32_t(j / kStages) & 1u, abort_flag)) {
              if (!*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 55); }
              *abort_flag = 1;
              break;
            }
            tc_fence_after();
            mma_stage(tmem, smem + s * kStageBytes, i > 0);
            mma_commit(&ctl.empty[s]);
            if (i == kBlockK / TK - 1) mma_commit(&ctl.tfull);
            committed = j + 1;
          }
        }
      }
    }
  } else {
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    int sums = 0;
    for (int it = blockIdx.x; it < items && !*abort_flag; it += gridDim.x) {
      const int r = (it / splits) * TM + q * 32 + lane;
      double acc[kCols];
#pragma unroll
      for (int u = 0; u < kCols; ++u) acc[u] = 0.0;
      for (int kb = first_block(it); kb < end_block(it); ++kb, ++sums) {
        const int ea = r < m ? __ldg(Ae + int64_t(kb) * m + r) : 0;
        // every wait ends in a warp vote, so a warp always leaves together (tcgen05.ld needs all 32 lanes)
        if (!__all_sync(0xffffffffu, mbar_wait(&ctl.tfull, uint32_t(sums) & 1u, abort_flag))) {
          if (lane == 0 && !*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, 56); }
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        long long v[kCols];
        const uint32_t fine = read_sums(tmem + lane_base + uint32_t(h * kCols), v);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.tempty);
        const int* be = Be + kb * TN + h * kCols;
#pragma unroll
        for (int u = 0; u < kCols; ++u)
          acc[u] = add_scaled<1>(acc[u], to_double(v[u], (fine >> u) & 1u), ea, __ldg(be + u));
      }
      if (r < m && !*abort_flag) {
        double2* dst = reinterpret_cast<double2*>(partial + (int64_t(it % splits) * m + r) * TN + h * kCols);
#pragma unroll
        for (int u = 0; u < kCols; u += 2) dst[u / 2] = make_double2(acc[u], acc[u + 1]);
      }
    }
  }

  __syncthreads();
  if (warp == 1) {
    if (ctl.abort_flag && lane == 0 && committed > 0) {
      // MMAs complete in order: once the last commit has arrived nothing reads tensor memory (bounded)
      const int jj = committed - 1;
      for (long long k = 0; k < (1 << 22); ++k) {
        if (mbar_try_wait(&ctl.empty[jj % kStages], uint32_t(jj / kStages) & 1u)) break;
        __nanosleep(64);
      }
    }
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// Digits of rows [r0, r0 + rows) of the m x n matrix, a warp per (row, 256-wide k block), 8 entries a lane: from FP64
// rows (A, lda, row 0 = row r0) or, with A null, from the sum of two FP32 planes.
__global__ void __launch_bounds__(256) matrix_digits_kernel(const double* __restrict__ A, const float* __restrict__ hi,
                                                            const float* __restrict__ lo, int64_t lda, int m, int n,
                                                            int nkb, int r0, int rows, uint16_t* __restrict__ Ad,
                                                            int* __restrict__ Ae) {
  const int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= int64_t(rows) * nkb) return;
  const int i = int(w / nkb), kb = int(w % nkb), k0 = kb * kBlockK + lane * 8;
  double v[8];
  int emax = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int64_t at = int64_t(i) * lda + k0 + u;
    v[u] = k0 + u < n ? (A ? A[at] : double(hi[at]) + double(lo[at])) : 0.0;
    emax = max(emax, exp_field(v[u]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  if (lane == 0) Ae[int64_t(kb) * m + r0 + i] = scale_exp(emax);
  const int64_t Kp = int64_t(nkb) * kBlockK;
  write_digits(v, emax, Ad + int64_t(r0 + i) * Kp + k0, int64_t(m) * Kp);
}

// Digits of X (n x R, ldx) as 64 columns (those from R on zero): a block per (k block, 8 columns), a warp a column.
__global__ void __launch_bounds__(256) columns_digits_kernel(const double* __restrict__ X, int64_t ldx, int n, int R,
                                                             int nkb, uint16_t* __restrict__ Bd,
                                                             int* __restrict__ Be, const int32_t* __restrict__ skip) {
  if (skip && *skip) return;
  __shared__ double t[kBlockK][9];
  const int kb = blockIdx.x, c0 = blockIdx.y * 8;
  for (int e = threadIdx.x; e < kBlockK * 8; e += blockDim.x) {
    const int k = e >> 3, c = c0 + (e & 7);
    t[k][e & 7] = (kb * kBlockK + k < n && c < R) ? X[int64_t(kb * kBlockK + k) * ldx + c] : 0.0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v[8];
  int emax = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    v[u] = t[lane * 8 + u][warp];
    emax = max(emax, exp_field(v[u]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  if (lane == 0) Be[kb * TN + c0 + warp] = scale_exp(emax);
  const int64_t Kp = int64_t(nkb) * kBlockK;
  write_digits(v, emax, Bd + int64_t(c0 + warp) * Kp + kb * kBlockK + lane * 8, TN * Kp);
}

// 3-D map over digit planes [7][rows][Kp] bf16, box 32 (k) x box_rows x 7, 64B swizzle
int make_map(CUtensorMap* map, void* base, int rows, int Kp, int box_rows) {
  cuuint64_t dims[3] = {cuuint64_t(Kp), cuuint64_t(rows), cuuint64_t(kDigits)};
  cuuint64_t strides[2] = {cuuint64_t(Kp) * 2, cuuint64_t(rows) * Kp * 2};
  cuuint32_t box[3] = {cuuint32_t(TK), cuuint32_t(box_rows), cuuint32_t(kDigits)};
  cuuint32_t estr[3] = {1, 1, 1};
  const EncodeTiledFn fn = encode_tiled();
  if (!fn) return UPDES_ERR_CUDA;
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? UPDES_OK : UPDES_ERR_CUDA;
}

size_t al256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

size_t ozaki64_scratch_bytes(int mmax, int ncmax, int Kmax) {
  const size_t Kp = size_t(ceil_div(Kmax, TK)) * TK;
  return al256(kDigits * size_t(mmax) * Kp * 2) + al256(kDigits * size_t(ncmax) * Kp * 2) + al256(size_t(mmax) * 4) +
         al256(size_t(ncmax) * 4) + 256;
}

int ozaki64_update(double* C, int64_t ldc, const double* A, int64_t lda, const double* B, int64_t ldb, int m, int nc,
                   int K, void* scratch, size_t scratch_bytes, DeviceStatus* st, cudaStream_t s, int max_ctas,
                   bool a_digits_ready, bool early) {
  if (m <= 0 || nc <= 0 || K <= 0) return UPDES_OK;
  if (K > 256) return UPDES_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < ozaki64_scratch_bytes(m, nc, K)) return UPDES_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(scratch) & 255) != 0) return UPDES_ERR_INVALID;
  const int Kp = int(ceil_div(K, TK)) * TK;
  // A's digits and exponents first: their place depends only on m and K, so an update with the same A can reuse them
  char* p = static_cast<char*>(scratch);
  uint16_t* Ad = reinterpret_cast<uint16_t*>(p);
  p += al256(kDigits * size_t(m) * Kp * 2);
  int* Ae = reinterpret_cast<int*>(p);
  p += al256(size_t(m) * 4);
  uint16_t* Bd = reinterpret_cast<uint16_t*>(p);
  p += al256(kDigits * size_t(nc) * Kp * 2);
  int* Be = reinterpret_cast<int*>(p);

  static std::atomic<unsigned long long> attr{0};
  if (int e = smem_opt_in((const void*)ozaki64_kernel, kSmemBytes, attr)) return e;
  CUtensorMap mapA, mapB;
  if (int e = make_map(&mapA, Ad, m, Kp, TM)) return e;
  if (int e = make_map(&mapB, Bd, nc, Kp, TN)) return e;
  StatScope sc(kStatGemm, s, 2.0 * m * double(nc) * K, double(m) * nc * 16.0 + (double(m) + nc) * K * 8.0);
  {
    int span = 1;
    while (span < Kp / 8) span *= 2;
    const int row_blocks = a_digits_ready ? 0 : int(ceil_div(int64_t(m) * span, 256));
    const int col_blocks = int(ceil_div(nc, 32 * (8 / (Kp / 32))));
    if (int e = launch_next(early && max_ctas == 0, digits64_kernel, unsigned(row_blocks + col_blocks), 256, 0, s, A, lda, m, B, ldb, nc, K, Kp,
                            span, row_blocks, Ad, Ae, Bd, Be))
      return e;
  }
  const int ntiles = int(ceil_div(m, TM) * ceil_div(nc, TN));
  const int grid = std::min(ntiles, max_ctas > 0 ? std::min(max_ctas, num_sms_cached()) : num_sms_cached());
  return launch_next(early, ozaki64_kernel, unsigned(grid), kThreads, kSmemBytes, s, mapA, mapB, Ae, Be, C, ldc, m, nc, Kp, st);
}

namespace {

struct MatrixDigits {
  uint16_t* d;
  int* e;
};
int k_blocks(int n) { return int(ceil_div(n, kBlockK)); }
MatrixDigits matrix_view(void* base, int rows, int n) {
  char* p = static_cast<char*>(base);
  return {reinterpret_cast<uint16_t*>(p),
          reinterpret_cast<int*>(p + al256(kDigits * size_t(rows) * k_blocks(n) * kBlockK * 2))};
}

}  // namespace

size_t rhs64_matrix_bytes(int m, int n) {
  return al256(kDigits * size_t(m) * k_blocks(n) * kBlockK * 2) + al256(size_t(m) * k_blocks(n) * 4);
}
size_t rhs64_columns_bytes(int n) { return rhs64_matrix_bytes(TN, n); }

// Row tiles times splits are dealt round robin to the SMs: the number of splits with the shortest longest share, a
// fraction of a block charged for writing and adding each split's sums.
int rhs64_splits(int m, int n) {
  const int tiles = int(ceil_div(m, TM)), nkb = k_blocks(n), sms = num_sms_cached();
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= std::min(nkb, kRhs64MaxSplits); ++s) {
    const double cost = double(ceil_div(int64_t(tiles) * s, sms) * ceil_div(nkb, s)) + 0.1 * s;
    if (cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

int rhs64_matrix(const double* A, const float* hi, const float* lo, int64_t lda, int m, int n, int r0, int rows,
                 void* matrix, cudaStream_t s) {
  const MatrixDigits v = matrix_view(matrix, m, n);
  matrix_digits_kernel<<<unsigned(ceil_div(int64_t(rows) * k_blocks(n) * 32, 256)), 256, 0, s>>>(
      A, hi, lo, lda, m, n, k_blocks(n), r0, rows, v.d, v.e);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}

int rhs64_setup() {
  static std::atomic<unsigned long long> attr{0};
  return smem_opt_in((const void*)rhs64_kernel, kStages * kStageBytes + 1024, attr);
}

int rhs64_multiply(const void* matrix, int m, int n, const double* X, int64_t ldx, int R, void* columns,
                   double* partial, int splits, DeviceStatus* st, cudaStream_t s, const int32_t* skip) {
  const int nkb = k_blocks(n);
  const MatrixDigits a = matrix_view(const_cast<void*>(matrix), m, n), b = matrix_view(columns, TN, n);
  CUtensorMap mapA, mapB;
  if (int e = make_map(&mapA, a.d, m, nkb * kBlockK, TM)) return e;
  if (int e = make_map(&mapB, b.d, TN, nkb * kBlockK, TN)) return e;
  if (int e = rhs64_setup()) return e;
  columns_digits_kernel<<<dim3(unsigned(nkb), TN / 8), 256, 0, s>>>(X, ldx, n, R, nkb, b.d, b.e, skip);
  UPDES_LAUNCH_CHECK();
  const int items = int(ceil_div(m, TM)) * splits;
  rhs64_kernel<<<std::min(items, num_sms_cached()), kThreads, kStages * kStageBytes + 1024, s>>>(
      mapA, mapB, a.e, b.e, partial, m, nkb, splits, st, skip);
  UPDES_LAUNCH_CHECK();
  return UPDES_OK;
}
