// Tensor-core trailing update of the mixed-precision LU, persistent and warp-specialised (sm_103a).
//
//   C  <-  C - A * B        C: FP32 hi/lo pairs ("double-float", ~48 bits)
//                           A: m x K FP32 (L factor block), B: K x nc FP32 (U factor block), K <= 256
//
// Numerics.  Every FP32 operand is written as 3 FP16 numbers under a power-of-two scale shared by a row of A (a
// column of B) over the whole K:
//   a = 2^(e-8) * (d0 + d1 + d2),  d0 an integer, |d0| <= 256;  d1 a multiple of 2^-12, |d1| <= 2^-1;  |d2| <= 2^-13,
// exact but for d2's rounding to 11 bits, at most 2^-33 of the row's maximum.  The products go to three FP32
// tensor-memory accumulators by their size: g0 = d0 e0, g1 = d0 e1 + d1 e0, g2 = d0 e2 + d1 e1 + d2 e0 + d1 e2 + d2 e1.
// The 256 products d0 e0 add up to an integer of at most 2^24: the tensor cores add no rounding to g0.  g1 is a multiple
// of 2^-12, exact up to 2^12.  It gets there only where the remainders behind the leading digits are alike over a row and a
// column: up to 2^16, where each of its 32 instructions drops 2^-8, 2^-32 of that sum's g0 (constant rows and columns lost
// all but 2^-26 of |A||B|).  Such rows and columns have their leading digits rounded at spread places instead
// (spread_place).  g2 is rounded below 2^-16 of its 2^8.  d2 e2 (2^-26,
// 2^-42 of the largest product) is left out: 8 products.  The epilogue forms g0 + g1 + g2 as a double-float with
// error-free transformations (FP32 ALU: GB300's FP64 rate is low) and subtracts it from C, once per tile.
// Measured against 64 bits, relative to |A||B|, K = 256, and beside it three 9-bit integer digits under a scale per 64 of
// K: normal entries 2^-37.8 (2^-29.1), columns graded by 2^-16 2^-32.8 (2^-27.6), cosines falling as 1/k 2^-33.1
// (2^-27.6), entries spread over 2^20 2^-29.6 (2^-23.9), within a factor of 4 2^-40.4 (2^-40.2), constant rows and columns
// 2^-32 (2^-36.4), 2^-10 of variation over a row 2^-31.  As a preconditioner the factors are the better for it: 7-8 iterations
// at n = 22,506 for 9-11.
// The small entries of a graded block matter to the Schur complement: with d1 cut at 2^-8 (g1 always exact) it took 14-25.
//
// What bounds it.  The previous form (tiles of 128 x 64, 8 products, a fold of four accumulators per 64 of K) moved 2.6 MB
// through shared memory for a 128 x 128 x 256 piece and took 25,600 clocks.  So the tiles are 128 x 128, the digit planes
// of B lie side by side so that one instruction of N = 256 forms d0 [e0 e1] in the neighbouring accumulators [g0 g1] and
// another d1 [e0 e1] in [g1 g2] (A is read once for two products), and one scale per K leaves one fold per tile: 1.8 MB,
// 15,400 clocks; 20,000 x 20,000 x 256 takes 1,310 us against 2,165.  Of these the products and the fold take 920 us without
// C, C's way (load, update, store, a warp after another) 1,390 without most products: the warps' chain over their pieces
// of C is what is left, with the tensor pipe 54 % and DRAM 60 % busy (n = 10,000).  C without an eviction hint: evict-first
// costs 10 %; neither prefetching C to L2 nor storing it from registers gains.
//
// Structure.  A pre-pass writes the digits once per update, laid out as the stages hold them, and the scales.  The main
// kernel is persistent (one CTA per SM, tiles of 128 x TN taken round robin) with three roles:
//   warp 0      producer: two bulk copies per 32 of K into a ring of stages (64B swizzle, 48 KB a stage);
//   warp 1      MMA issuer: 6 instructions of tcgen05.mma (kind::f16, M=128) per 16 of K into the three accumulators
//               of TN columns each;
//   warps 2-9   epilogue, a 32-row x TN/2-column piece of the tile each: tcgen05.ld, fold, then C -= acc on 32 columns
//               at a time in the warp's own buffer, which its first lane loads and stores by TMA.
// There is one accumulator set (384 of the 512 TMEM columns).  The last stage of a tile issues g0's and g1's products first
// and commits them, so that the epilogue reads them while g2's run; the next tile's first instructions only wait
// for those.  The fold and the C traffic run beside the next tile's MMAs.  Every mbarrier wait is bounded; a
// timeout sets the status word and an abort flag that every role checks, and tensor memory is freed on every path.
#include <atomic>

#include <cuda_fp16.h>

#include "gemm_tc.cuh"
#include "stats.cuh"
#include "tc.cuh"

namespace {

constexpr int TM = 128, TK = 32;
constexpr int kMaxK = 256;   // one exact accumulation
constexpr int kKpUnit = 64;  // K is padded to this
constexpr int kDigits = 3, kGroups = 3;
constexpr int kEpiWarps = 8;
constexpr int kWarps = 2 + kEpiWarps, kThreads = kWarps * 32;
constexpr uint32_t kTmemCols = 512;
constexpr int kATile = TM * TK * 2;           // 8 KB per digit plane
constexpr int kCBox = 32 * 32 * 4;            // 32 rows x 32 FP32 (128-byte rows): 4 KB
constexpr int kCBytes = kEpiWarps * 2 * kCBox;  // {hi, lo} per epilogue warp

template <int TN>
struct Cfg {
  static constexpr int kStages = TN == 128 ? 3 : 4;
  static constexpr int kBTile = TN * TK * 2;
  static constexpr int kStageBytes = kDigits * (kATile + kBTile);  // 48 KB (TN = 64: 36 KB)
  static constexpr int kSmemBytes = kStages * kStageBytes + kCBytes + 1024;
  static constexpr int kCols = TN / 2;  // columns of an epilogue warp
  static_assert(kSmemBytes <= 227 * 1024, "shared memory");
  static_assert(kGroups * TN <= int(kTmemCols), "tensor memory");
};

// instruction descriptor: D = F32, A = B = F16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc(int n) {
  return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(TM >> 4) << 24);
}

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

__device__ __forceinline__ int exp_of(float mx) {
  const int E = (__float_as_int(mx) >> 23) & 0xFF;
  if (E == 0) return -100;
  return max(E - 126, -100);
}

// Error-free sum (Knuth's TwoSum) and Dekker's Fast2Sum on column pairs, with the packed FP32x2 instructions
// of sm_100+ (one issue slot per pair).  y - x is formed as fma(x, -1, y): the product is exact, so it rounds once like a subtraction.
__device__ __forceinline__ float2 sub2(float2 y, float2 x) { return __ffma2_rn(x, make_float2(-1.f, -1.f), y); }

__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
  s = __fadd2_rn(a, b);
  const float2 bb = sub2(s, a);
  e = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}

__device__ __forceinline__ void fast_two_sum2(float2 a, float2 b, float2& s, float2& e) {
  s = __fadd2_rn(a, b);
  e = sub2(b, sub2(s, a));
}

// A row or column in whose runs of 64 steps the remainders behind the leading digits add up to more than this in all (in
// units of that digit, with the entries' signs; without a pattern 7 +- 3) hardly varies: its d1 are alike, and sums with
// another such one outgrow g1's 24 bits.  Its leading digits are rounded at places spread over the steps instead, which
// lets the remainders cancel and takes d2 a bit.
constexpr int kAlike = 24 << 12;  // in units of 2^-12
__device__ __forceinline__ int remainder_of(float v, float scale) {
  const float x = fabsf(__fmul_rn(v, scale));
  return __float2int_rn(__fmul_rn(__fsub_rn(x, rintf(x)), 4096.f));
}
// The warp's largest of numbers that are not negative.
__device__ __forceinline__ float warp_max(float v) {
  return __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(v)));
}
// The k-th place, between -1/2 and 1/2: the fraction of k times the golden ratio, spread evenly over any run of steps and,
// unlike the bits of k in reverse, over every other or every third step too, where signs may alternate.
__device__ __forceinline__ float spread_place(int k) {
  return float(int(unsigned(k) * 0x9E3779B9u)) * 0x1p-32f;
}

// The digits of one FP32 value under `scale` (|v * scale| < 256), the leading one rounded with `place` added: every step is
// exact but the last conversion.
__device__ __forceinline__ void split3(float v, float scale, float place, float (&d)[kDigits]) {
  const float x = __fmul_rn(v, scale);
  d[0] = copysignf(rintf(__fadd_rn(fabsf(x), place)), x);
  const float y = __fmul_rn(__fsub_rn(x, d[0]), 4096.f);
  // |y| <= 2048, or 4096 with a place: 11 bits and a sign, exact in FP16 (beyond 2048 the even ones)
  const float i1 = __half2float(__float2half_rn(rintf(y)));
  d[1] = __fmul_rn(i1, 0x1p-12f);
  d[2] = __fmul_rn(__fsub_rn(y, i1), 0x1p-12f);
}

// Digits lie as the stages of the main kernel hold them: for each tile of `rows` rows (columns of B) and each 32 of K
// one contiguous piece [plane][row][32], with 64-byte rows in the 64B swizzle (16-byte chunk c of row r at c ^ ((r >> 1) & 3)).
// Element offset of (row r of tile t, k) in plane p.
__device__ __forceinline__ int64_t digit_at(int64_t t, int r, int p, int k, int nks, int rows) {
  return ((t * nks + k / TK) * kDigits + p) * int64_t(rows * TK) + r * TK + ((((k % TK) >> 3) ^ ((r >> 1) & 3)) << 3) + (k & 7);
}

// `NK` k-steps of 16 from one stage for operands A and B (descriptors of their first rows): D (+)= A B.  Descriptors
// are built once per stage; every operand offset is a compile-time constant added to them (address units of 16 bytes).
template <int NK, bool FIRST>
__device__ __forceinline__ void mma_steps(uint32_t d, uint64_t a0, uint64_t b0, uint32_t id) {
#pragma unroll
  for (int kk = 0; kk < NK; ++kk) {
    if (FIRST && kk == 0) mma_bf16<false>(d, a0, b0, id);  // kind::f16: the descriptor says FP16
    else mma_bf16<true>(d, a0 + uint64_t(kk * 2), b0 + uint64_t(kk * 2), id);
  }
}

// ---- digit pre-pass ------------------------------------------------------------------------------------
// The digits of row r of tile t (`rows` rows a tile): v[u][w] is the entry k = 64 u + 2 lane + w.
__device__ __forceinline__ void write_digits(const float (&v)[kMaxK / 64][2], float scale, int lane, int Kp, int64_t t, int r,
                                             int rows, __half* __restrict__ out) {
  int left = 0;
#pragma unroll
  for (int u = 0; u < kMaxK / 64; ++u)
    left += abs(__reduce_add_sync(0xffffffffu, remainder_of(v[u][0], scale) + remainder_of(v[u][1], scale)));
  const bool alike = left > kAlike;
#pragma unroll
  for (int u = 0; u < kMaxK / 64; ++u) {
    if (u * 64 >= Kp) break;
    const int k = u * 64 + 2 * lane;
    float da[kDigits], db[kDigits];
    split3(v[u][0], scale, alike ? spread_place(k) : 0.f, da);
    split3(v[u][1], scale, alike ? spread_place(k + 1) : 0.f, db);
#pragma unroll
    for (int p = 0; p < kDigits; ++p)
      *reinterpret_cast<__half2*>(out + digit_at(t, r, p, k, Kp / TK, rows)) = __floats2half2_rn(da[p], db[p]);
  }
}

// A (m x K, lda) -> Ad (see digit_at) and As[r] = 2^(e-8), one warp per row; bx is the block's index among the row
// part's blocks.
__device__ __forceinline__ void digits_rows(int bx, const float* A, int64_t lda, int m, int K, int Kp,
                                            __half* __restrict__ Ad, float* __restrict__ As) {
  const int64_t r = (int64_t(bx) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= m) return;
  float v[kMaxK / 64][2];
  float mx = 0.f;
#pragma unroll
  for (int u = 0; u < kMaxK / 64; ++u)
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int k = u * 64 + 2 * lane + w;
      v[u][w] = k < K ? A[r * lda + k] : 0.f;
      mx = fmaxf(mx, fabsf(v[u][w]));
    }
  mx = warp_max(mx);
  const int e = exp_of(mx);
  if (lane == 0) As[r] = pow2f(e - 8);
  write_digits(v, pow2f(8 - e), lane, Kp, r / TM, int(r % TM), TM, Ad);
}

// B (K x nc, ldb) -> Bd (transposed, in tiles of TN columns) and Bs[c]; a CTA per 32 columns.
__device__ __forceinline__ void digits_cols(int bx, const float* B, int64_t ldb, int nc, int K, int Kp, int TN,
                                            __half* __restrict__ Bd, float* __restrict__ Bs) {
  __shared__ float t[kMaxK][33];
  const int c0 = bx * 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 16  // loads in flight together: the pass is short and mostly their latency
  for (int k = warp; k < Kp; k += 8)
    t[k][lane] = (k < K && c0 + lane < nc) ? B[int64_t(k) * ldb + c0 + lane] : 0.f;
  __syncthreads();
  for (int c = warp; c < 32; c += blockDim.x / 32) {
    const int64_t gc = c0 + c;
    if (gc >= nc) continue;
    float v[kMaxK / 64][2];
    float mx = 0.f;
#pragma unroll
    for (int u = 0; u < kMaxK / 64; ++u)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        v[u][w] = u * 64 < Kp ? t[u * 64 + 2 * lane + w][c] : 0.f;
        mx = fmaxf(mx, fabsf(v[u][w]));
      }
    mx = warp_max(mx);
    const int e = exp_of(mx);
    if (lane == 0) Bs[gc] = pow2f(e - 8);
    write_digits(v, pow2f(8 - e), lane, Kp, gc / TN, int(gc % TN), TN, Bd);
  }
}

// Both digit passes of one update in a single launch: blocks [0, row_blocks) take the rows of A, the others the
// column tiles of B.
__global__ void __launch_bounds__(256) digits_kernel(const float* A, int64_t lda, int m, const float* B, int64_t ldb, int nc, int K, int Kp,
                                                     int TN, int row_blocks, __half* __restrict__ Ad, float* __restrict__ As,
                                                     __half* __restrict__ Bd, float* __restrict__ Bs) {
  const int b = int(blockIdx.x);
  allow_next();
  wait_previous();
  if (b < row_blocks) digits_rows(b, A, lda, m, K, Kp, Ad, As);
  else digits_cols(b - row_blocks, B, ldb, nc, K, Kp, TN, Bd, Bs);
}

// ---- main kernel ---------------------------------------------------------------------------------------
struct Ctrl {
  uint64_t full[4], empty[4];  // operand stages: filled by TMA / their MMAs are done
  uint64_t hi_done, lo_done;   // the tile's g0 and g1 / g2 are complete
  uint64_t hi_free, lo_free;   // every epilogue warp has read them
  uint64_t cfull[kEpiWarps];   // a warp's piece of C has arrived
  uint32_t tmem;
  int abort_flag;
};

// A contiguous copy into shared memory that completes on an mbarrier (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

template <int TN>
__global__ void __launch_bounds__(kThreads, 1)
    ozaki3_kernel(const __grid_constant__ CUtensorMap tmCh, const __grid_constant__ CUtensorMap tmCl,
                  const __half* Ad, const __half* Bd, const float* As, const float* Bs, int m, int nc, int Kp,
                  DeviceStatus* st) {
  using C = Cfg<TN>;
  constexpr int kStages = C::kStages, kBTile = C::kBTile, kStageBytes = C::kStageBytes, kCols = C::kCols;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ Ctrl ctl;
  __shared__ __align__(16) float s_scales[kEpiWarps][kCols];  // of a warp's columns of B
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_n = int(ceil_div(nc, TN)), tiles_m = int(ceil_div(m, TM));
  const int ntiles = tiles_n * tiles_m;
  const int nks = Kp / TK;  // at least 2
  volatile int* abort_flag = &ctl.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 1);
    }
    mbar_init(&ctl.hi_done, 1);
    mbar_init(&ctl.lo_done, 1);
    mbar_init(&ctl.hi_free, kEpiWarps);
    mbar_init(&ctl.lo_free, kEpiWarps);
    for (int w = 0; w < kEpiWarps; ++w) mbar_init(&ctl.cfull[w], 1);
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
  int last_commit = -1;  // MMA issuer: index of the last committed stage
  auto give_up = [&](int tag) {
    if (!*abort_flag) { status_error(st, UPDES_ERR_TIMEOUT); atomicCAS(&st->timeout_tag, 0, tag); }
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint64_t pol_keep = l2_policy_evict_last();
      int j = 0;
      for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
        const uint8_t* gA = reinterpret_cast<const uint8_t*>(Ad) + int64_t(t / tiles_n) * nks * (kDigits * kATile);
        const uint8_t* gB = reinterpret_cast<const uint8_t*>(Bd) + int64_t(t % tiles_n) * nks * (kDigits * kBTile);
        for (int ks = 0; ks < nks; ++ks, ++j) {
          const int s = j % kStages;
          if (!mbar_wait(&ctl.empty[s], (uint32_t(j / kStages) & 1u) ^ 1u, abort_flag)) {
            give_up(41);
            break;
          }
          uint8_t* sA = smem + s * kStageBytes;
          mbar_expect_tx(&ctl.full[s], uint32_t(kStageBytes));
          bulk_load(smem_u32(sA), gA + ks * (kDigits * kATile), kDigits * kATile, &ctl.full[s], pol_keep);
          bulk_load(smem_u32(sA + kDigits * kATile), gB + ks * (kDigits * kBTile), kDigits * kBTile, &ctl.full[s], pol_keep);
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
      constexpr int NK = TK / 16;
      constexpr uint32_t id1 = idesc(TN), id2 = idesc(2 * TN);
      const uint32_t g01 = tmem, g12 = tmem + uint32_t(TN), g2 = tmem + uint32_t(2 * TN);
      int j = 0, tl = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok && !*abort_flag; t += gridDim.x, ++tl) {
        for (int ks = 0; ks < nks; ++ks, ++j) {
          const int s = j % kStages;
          ok = mbar_wait(&ctl.full[s], uint32_t(j / kStages) & 1u, abort_flag) &&
               (ks != 0 || mbar_wait(&ctl.hi_free, (uint32_t(tl) & 1u) ^ 1u, abort_flag));
          if (!ok) {
            give_up(42);
            break;
          }
          tc_fence_after();
          const uint8_t* sA = smem + s * kStageBytes;
          const uint64_t a0 = make_desc(smem_u32(sA)), a1 = a0 + uint64_t(kATile >> 4), a2 = a0 + uint64_t(2 * (kATile >> 4));
          const uint64_t b0 = make_desc(smem_u32(sA + kDigits * kATile)), b1 = b0 + uint64_t(kBTile >> 4),
                         b2 = b0 + uint64_t(2 * (kBTile >> 4));
          if (ks == 0) {
            mma_steps<NK, true>(g01, a0, b0, id2);  // d0 [e0 e1] -> [g0 g1]
            ok = mbar_wait(&ctl.lo_free, (uint32_t(tl) & 1u) ^ 1u, abort_flag);
            if (ok) {
              tc_fence_after();
              mma_steps<NK, true>(g2, a0, b2, id1);    // d0 e2 -> g2
              mma_steps<NK, false>(g12, a1, b0, id2);  // d1 [e0 e1] -> [g1 g2]
              mma_steps<NK, false>(g2, a1, b2, id1);   // d1 e2 -> g2
              mma_steps<NK, false>(g2, a2, b0, id1);   // d2 e0 -> g2
              mma_steps<NK, false>(g2, a2, b1, id1);   // d2 e1 -> g2
            }
          } else {
            mma_steps<NK, false>(g01, a0, b0, id2);
            mma_steps<NK, false>(g12, a1, b0, id2);
            if (ks == nks - 1) mma_commit(&ctl.hi_done);
            mma_steps<NK, false>(g2, a0, b2, id1);
            mma_steps<NK, false>(g2, a1, b2, id1);
            mma_steps<NK, false>(g2, a2, b0, id1);
            mma_steps<NK, false>(g2, a2, b1, id1);
            if (ks == nks - 1) mma_commit(&ctl.lo_done);
          }
          mma_commit(&ctl.empty[s]);
          last_commit = j;
          if (!ok) {
            give_up(44);
            break;
          }
        }
      }
    }
  } else {
    // ---------------- epilogue: lane quarter q = warp % 4, column group h ----------------
    const int q = warp & 3, h = (warp - 2) >> 2, ew = warp - 2;
    const uint64_t pol_c = l2_policy_unchanged();
    uint8_t* bufh = smem + kStages * kStageBytes + ew * 2 * kCBox;
    uint8_t* bufl = bufh + kCBox;
    uint64_t* cbar = &ctl.cfull[ew];
    float* scales = s_scales[ew];
    const uint32_t lane_base = (uint32_t(q * 32) << 16) + uint32_t(h * kCols);
    int loads = 0, waited = 0;  // pieces of C requested / taken over
    // the warp's pieces of C, 32 columns each, in the order in which it takes them: (tile, slice), those inside C only
    auto piece_in = [&](int t, int sl) {
      return t < ntiles && (t / tiles_n) * TM + q * 32 < m && (t % tiles_n) * TN + h * kCols + sl * 32 < nc;
    };
    auto load_c = [&](int t, int sl) {
      const int y = (t / tiles_n) * TM + q * 32, x = (t % tiles_n) * TN + h * kCols + sl * 32;
      if (lane == 0) {
        mbar_expect_tx(cbar, uint32_t(2 * kCBox));
        tma_load_2d(smem_u32(bufh), &tmCh, x, y, cbar, pol_c);
        tma_load_2d(smem_u32(bufl), &tmCl, x, y, cbar, pol_c);
      }
      ++loads;
    };
    auto load_first = [&](int t) {  // of tile t or the next of the CTA's tiles in which the warp has one
      while (t < ntiles && !piece_in(t, 0)) t += int(gridDim.x);
      if (t < ntiles) load_c(t, 0);
    };
    load_first(int(blockIdx.x));
    int tl = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++tl) {
      const int r0 = (t / tiles_n) * TM + q * 32, c0 = (t % tiles_n) * TN + h * kCols;
      const uint32_t ph = uint32_t(tl) & 1u;
      const float sa = r0 + lane < m ? -__ldcg(As + r0 + lane) : 0.f;
      // the columns' scales, for every lane (those of columns beyond nc are scratch bytes of no effect: the store leaves
      // these columns out)
      __syncwarp();
#pragma unroll
      for (int u = lane; u < kCols; u += 32) scales[u] = __ldcg(Bs + c0 + u);
      float2 gh[kCols / 2], gl[kCols / 2];  // the row's sums over the warp's columns, as column pairs
      // every wait ends in a warp vote, so a warp always leaves together (tcgen05.ld needs all 32 lanes)
      if (!__all_sync(0xffffffffu, mbar_wait(&ctl.hi_done, ph, abort_flag))) {
        if (lane == 0) give_up(43);
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < kCols / 2; u += 8) {
        tmem_ld16(tmem + lane_base + uint32_t(2 * u), reinterpret_cast<float*>(gh + u));
        tmem_ld16(tmem + lane_base + uint32_t(TN + 2 * u), reinterpret_cast<float*>(gl + u));
      }
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.hi_free);
#pragma unroll
      for (int u = 0; u < kCols / 2; ++u) {
        float2 s, e;
        two_sum2(gh[u], gl[u], s, e);
        gh[u] = s;
        gl[u] = e;
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&ctl.lo_done, ph, abort_flag))) {
        if (lane == 0) give_up(47);
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < kCols / 2; u += 8) {
        float2 g[8];
        tmem_ld16(tmem + lane_base + uint32_t(2 * TN + 2 * u), reinterpret_cast<float*>(g));
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) gl[u + i] = __fadd2_rn(gl[u + i], g[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.lo_free);
      // ---- C -= sums, 32 columns at a time ----
      bool ok = true;
#pragma unroll
      for (int sl = 0; sl < kCols / 32; ++sl) {
        if (!ok || !piece_in(t, sl)) continue;
        const float4* sb = reinterpret_cast<const float4*>(scales + sl * 32);
        ok = __all_sync(0xffffffffu, mbar_wait(cbar, uint32_t(waited) & 1u, abort_flag));
        if (!ok) {
          if (lane == 0) give_up(45);
          continue;
        }
        ++waited;
        // the lane's row in the 128B-swizzled boxes: 16-byte chunk c of row r sits at chunk c ^ (r & 7)
        uint8_t* hrow = bufh + lane * 128;
        uint8_t* lrow = bufl + lane * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int off = ((c ^ (lane & 7)) << 4);
          const float4 sb4 = sb[c];
          const float4 hv = *reinterpret_cast<float4*>(hrow + off), lv = *reinterpret_cast<float4*>(lrow + off);
          float2 hx[2] = {make_float2(hv.x, hv.y), make_float2(hv.z, hv.w)};
          float2 lx[2] = {make_float2(lv.x, lv.y), make_float2(lv.z, lv.w)};
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int pi = sl * 16 + c * 2 + u;
            // minus the product of the scales, a power of two: exact
            const float2 sc = __fmul2_rn(make_float2(sa, sa), u ? make_float2(sb4.z, sb4.w) : make_float2(sb4.x, sb4.y));
            float2 sx, tx;
            two_sum2(hx[u], __fmul2_rn(gh[pi], sc), sx, tx);
            tx = __fadd2_rn(tx, __ffma2_rn(gl[pi], sc, lx[u]));
            fast_two_sum2(sx, tx, hx[u], lx[u]);
          }
          *reinterpret_cast<float4*>(hrow + off) = make_float4(hx[0].x, hx[0].y, hx[1].x, hx[1].y);
          *reinterpret_cast<float4*>(lrow + off) = make_float4(lx[0].x, lx[0].y, lx[1].x, lx[1].y);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic accesses before TMA's
        __syncwarp();
        if (lane == 0) {
          // rows >= m and columns >= nc are outside the tensor and are not written
          tma_store_2d(&tmCh, c0 + sl * 32, r0, smem_u32(bufh), pol_c);
          tma_store_2d(&tmCl, c0 + sl * 32, r0, smem_u32(bufl), pol_c);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the buffer has been read
        }
        // the warp's next piece: the tile's next slice or the first one of a later tile
        if (sl + 1 < kCols / 32 && piece_in(t, sl + 1)) {
          load_c(t, sl + 1);
        } else {
          load_first(t + int(gridDim.x));
        }
      }
      if (!ok) break;
    }
    if (lane == 0) {
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // stores complete before exit
      if (loads > waited) {
        // a C load still in flight (only after an abort) must land before shared memory goes away (bounded)
        for (long long it = 0; it < (1 << 22); ++it) {
          if (mbar_try_wait(cbar, uint32_t(waited) & 1u)) break;
          __nanosleep(64);
        }
      }
    }
    __syncwarp();
  }

  // ---- teardown: all roles done; make sure no MMA is in flight before tensor memory is freed ----
  __syncthreads();
  if (warp == 1) {
    if (ctl.abort_flag && lane == 0 && last_commit >= 0) {
      // MMAs complete in order: once the last commit has arrived nothing reads tensor memory (bounded)
      for (long long it = 0; it < (1 << 22); ++it) {
        if (mbar_try_wait(&ctl.empty[last_commit % kStages], uint32_t(last_commit / kStages) & 1u)) break;
        __nanosleep(64);
      }
    }
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// 2-D map over an FP32 plane (rows x cols, row stride ld elements), box 32 columns x 32 rows, 128B swizzle
int make_map_c(CUtensorMap* map, float* base, int rows, int cols, int64_t ld) {
  const EncodeTiledFn fn = encode_tiled();
  if (!fn) return UPDES_ERR_CUDA;
  cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(ld) * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? UPDES_OK : UPDES_ERR_CUDA;
}

template <int TN>
int launch_update(const CUtensorMap (&maps)[2], const __half* Ad, const __half* Bd, const float* As, const float* Bs, int m, int nc, int Kp, int ctas,
                  DeviceStatus* st, cudaStream_t s, bool early) {
  static std::atomic<unsigned long long> attr{0};
  if (int e = smem_opt_in((const void*)ozaki3_kernel<TN>, Cfg<TN>::kSmemBytes, attr)) return e;
  const int64_t ntiles = ceil_div(m, TM) * ceil_div(nc, TN);
  return launch_next(early, ozaki3_kernel<TN>, unsigned(std::min<int64_t>(ntiles, ctas)), kThreads, Cfg<TN>::kSmemBytes, s,
                     maps[0], maps[1], Ad, Bd, As, Bs, m, nc, Kp, st);
}

}  // namespace

size_t ozaki3_scratch_bytes(int mmax, int ncmax, int Kmax) {
  const size_t Kp = size_t(ceil_div(Kmax, kKpUnit)) * kKpUnit;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t mp = size_t(ceil_div(mmax, TM)) * TM, ncp = size_t(ceil_div(ncmax, 128)) * 128;  // whole tiles
  return al(kDigits * mp * Kp * 2) + al(kDigits * ncp * Kp * 2) + al(mp * 4) + al(ncp * 4) + 256;
}

int ozaki3_update(float* Chi, float* Clo, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb,
                  int m, int nc, int K, void* scratch, size_t scratch_bytes, DeviceStatus* st, cudaStream_t s,
                  int max_ctas, bool a_digits_ready, bool early) {
  if (m <= 0 || nc <= 0 || K <= 0) return UPDES_OK;
  if (K > kMaxK) return UPDES_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < ozaki3_scratch_bytes(m, nc, K)) return UPDES_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(scratch) & 255) != 0) return UPDES_ERR_INVALID;
  // C goes through TMA: 16-byte aligned planes and row stride (else the caller uses the other kernel)
  if (((reinterpret_cast<uintptr_t>(Chi) | reinterpret_cast<uintptr_t>(Clo)) & 15) != 0 || (ldc & 3) != 0)
    return UPDES_ERR_UNSUPPORTED;
  const int Kp = int(ceil_div(K, kKpUnit)) * kKpUnit;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  // A's digits and scales first: their place depends only on m and K, so an update with the same A can reuse them
  const size_t mp = size_t(ceil_div(m, TM)) * TM, ncp = size_t(ceil_div(nc, 128)) * 128;
  char* p = static_cast<char*>(scratch);
  __half* Ad = reinterpret_cast<__half*>(p);
  p += al(kDigits * mp * Kp * 2);
  float* As = reinterpret_cast<float*>(p);
  p += al(mp * 4);
  __half* Bd = reinterpret_cast<__half*>(p);
  p += al(kDigits * ncp * Kp * 2);
  float* Bs = reinterpret_cast<float*>(p);

  const int ctas = max_ctas > 0 ? std::min(max_ctas, num_sms_cached()) : num_sms_cached();
  // Tiles of 128 columns unless tiles of 64, which take about 0.55 of their time, finish in fewer rounds for it: with at
  // most one tile a CTA (1,000 x 1,000 x 256: 21 us against 25), or where much of the last 128 columns is empty
  // (20,000 x 192 x 64: 30 against 35).  With many rounds the wide tiles win (3,000 x 3,000 x 256: 49 against 59).
  const int64_t rows = ceil_div(m, TM), w128 = ceil_div(rows * ceil_div(nc, 128), ctas),
                w64 = ceil_div(rows * ceil_div(nc, 64), ctas);
  const bool wide = 9 * w128 <= 5 * w64;
  CUtensorMap maps[2];
  int e = make_map_c(&maps[0], Chi, m, nc, ldc);
  if (e) return e;
  if ((e = make_map_c(&maps[1], Clo, m, nc, ldc))) return e;

  StatScope sc(kStatGemm, s, 2.0 * m * double(nc) * K, double(m) * nc * 16.0 + (double(m) + nc) * K * 4.0);
  const int row_blocks = a_digits_ready ? 0 : int(ceil_div(int64_t(m) * 32, 256));
  if ((e = launch_next(early && max_ctas == 0, digits_kernel, unsigned(row_blocks + ceil_div(nc, 32)), 256, 0, s, A, lda, m, B, ldb, nc, K, Kp,
                       wide ? 128 : 64, row_blocks, Ad, As, Bd, Bs)))
    return e;
  return wide ? launch_update<128>(maps, Ad, Bd, As, Bs, m, nc, Kp, ctas, st, s, early)
              : launch_update<64>(maps, Ad, Bd, As, Bs, m, nc, Kp, ctas, st, s, early);
}
