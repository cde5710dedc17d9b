// LU panel on one thread-block cluster: the panel's rows live in registers, a row (or up to six) per thread, and
// the per-column pivot exchange goes through distributed shared memory.
//
// What bounds it.  A panel is a chain of `nb` columns, each a maximum over all rows and an update that needs its
// winner, so its time is nb times the latency of one column.  Between the CTAs of a grid that exchange costs two
// trips through L2 (a record published and polled, then the winner's row fetched).  Inside a cluster every CTA
// pushes its candidate, row and all, into the shared memory of every other (st.async, completing on the
// receiver's mbarrier): one trip, no polling of global memory, no fetch.  The push costs about 280 cycles to one
// CTA and grows with the bytes (16 CTAs of 256 bytes to each other: about 1,000), so the cluster is the smallest
// that holds the rows (one CTA up to 768 rows of 64 floats: no exchange at all), and only the columns that are
// still to be eliminated travel.
//
// Rows never move.  A row's place in the interchanged panel is a number its thread keeps: the pivot's thread
// takes the diagonal's number, the thread that had it takes the pivot's, and the places are applied when the
// panel is written back.  The columns left of a row shift down by one register with every step (the update writes
// entry i to i - 1), so every register index is a constant; a multiplier goes to shared memory as it is made.
// Per column: wait for the candidates, pick (largest |a|, smallest place on ties), scale, update, search
// column j + 1 on the way, CTA maximum, and the winner's warp publishes its row: one CTA barrier (two in a
// one-CTA cluster, which has no other hand-over).
//
// Beyond 12,288 rows of 64 floats (three a thread in 16 CTAs) a thread keeps up to six rows, half of the columns at a
// time: the left 32 are eliminated, the pivots' rows of the right half are solved for in every CTA, each thread applies
// the 32 multipliers to its rows of the right half where they lie, in the elimination's order, and that half follows.  135
// us at 12,300 rows, 170 at 20,000, 217 at 22,500 (its update is plain arithmetic, its exchanges carry half the bytes),
// where CTAs that meet in L2 took about 260.
//
// Receive slots rotate over three columns: a CTA publishes column j + 3 into column j's slot only after it has
// every candidate of column j + 2, and each CTA publishes that one after it is done with column j.
// Waits are bounded; a CTA that gives up records a timeout, and all CTAs of the cluster meet at a last barrier
// before any of them leaves, so no store goes to a CTA that has left.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "lu.cuh"
#include "stats.cuh"

namespace {

constexpr int kThreads = 256, kW = kThreads / 32;
constexpr int kMaxC = 16;   // CTAs of a cluster (16 needs the non-portable attribute)
constexpr int kSlots = 3;
constexpr int kMaxRows = 3;  // rows a thread can hold: 3 x 64 floats or 3 x 32 doubles in registers
constexpr uint32_t kNoRow = 0x7fffffffu;

// Columns of a panel: 256 bytes of a row either way (FP64 panels are bound by the SM's two FP64 multiply-adds a
// cycle, half as many columns halve that work per row).
template <typename T>
constexpr int kCols = 256 / int(sizeof(T));

// A candidate: its order key, its row's place, 1 / pivot and the row's entries in the columns from the current one on.
template <typename T>
struct alignas(16) Rec {
  uint4 head;       // key (one or two words), place
  T rinv[16 / sizeof(T)];
  T row[kCols<T>];
};

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void push16(uint32_t dst, uint4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool phase_done(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Order key of |a|: 0 for "no candidate", else the bits of |a| + 1 (NaN as infinity, so that it surfaces as a
// bad pivot), which order like the values.
__device__ __forceinline__ uint32_t key_of(float a) {
  return min(__float_as_uint(a) & 0x7fffffffu, 0x7f800000u) + 1u;
}
__device__ __forceinline__ unsigned long long key_of(double a) {
  return min(static_cast<unsigned long long>(__double_as_longlong(a)) & 0x7fffffffffffffffull,
             0x7ff0000000000000ull) + 1ull;
}
__device__ __forceinline__ bool usable(uint32_t key) { return key > 1u && key <= 0x7f800000u; }
__device__ __forceinline__ bool usable(unsigned long long key) { return key > 1ull && key <= 0x7ff0000000000000ull; }
// The warp's largest key and, of the lanes that hold it, the smallest row (kNoRow if every key is 0).  Reductions by
// all lanes, in a fixed order: no vote, no branch.
__device__ __forceinline__ void warp_best(uint32_t& key, uint32_t& row) {
  const uint32_t km = __reduce_max_sync(0xffffffffu, key);
  row = __reduce_min_sync(0xffffffffu, key == km ? row : kNoRow);
  key = km;
}
__device__ __forceinline__ void warp_best(unsigned long long& key, uint32_t& row) {
  const uint32_t hi = uint32_t(key >> 32), lo = uint32_t(key);
  const uint32_t hm = __reduce_max_sync(0xffffffffu, hi);
  const uint32_t lm = __reduce_max_sync(0xffffffffu, hi == hm ? lo : 0u);
  row = __reduce_min_sync(0xffffffffu, (hi == hm && lo == lm) ? row : kNoRow);
  key = (static_cast<unsigned long long>(hm) << 32) | lm;
}
__device__ __forceinline__ uint4 put_head(uint32_t key, uint32_t row) { return make_uint4(key, 0u, row, 0u); }
__device__ __forceinline__ uint4 put_head(unsigned long long key, uint32_t row) {
  return make_uint4(uint32_t(key), uint32_t(key >> 32), row, 0u);
}
__device__ __forceinline__ void get_key(uint4 h, uint32_t& key) { key = h.x; }
__device__ __forceinline__ void get_key(uint4 h, unsigned long long& key) {
  key = (static_cast<unsigned long long>(h.y) << 32) | h.x;
}
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename T>
constexpr int fixed_bytes() {
  return (kSlots * kMaxC + 2) * int(sizeof(Rec<T>));
}
template <typename T>
constexpr int lds_of(int rows) { return rows | 1; }  // odd row stride of the multipliers: no bank conflicts either way
template <typename T>
size_t smem_bytes(int rows, int nbh, int halves) {  // nbh columns at a time, in one or two halves
  return fixed_bytes<T>() + size_t(nbh) * lds_of<T>(rows) * sizeof(T) + (halves == 2 ? 2 * nbh * (nbh + 1) * sizeof(T) : 0);
}

template <int V>
struct Int { static constexpr int value = V; };

// Factors W[k:n, k:k+nb] in place, NB columns at a time: all of them (H = 1, nb <= NB), or the left half, then the
// right half's update, then the right half (H = 2, nb = 2 NB).  piv[k..k+nb): the interchanges; swap_map (may be null): [0] count,
// [1..128] destination rows, [129..256] source rows of their net permutation.
template <typename T, int R, int NB, int H>
__global__ void __launch_bounds__(kThreads, 1)
    panel_cluster_kernel(T* W, int64_t ld, int n, int k, int nb, int rows_per_cta, int32_t* __restrict__ piv,
                         int32_t* swap_map, DeviceStatus* st) {
  using Key = decltype(key_of(T(0)));
  constexpr int kElems = 16 / int(sizeof(T));
  constexpr int kHeads = 2;  // 16-byte words before the row
  extern __shared__ __align__(16) unsigned char pc_smem[];
  Rec<T>(*recv)[kMaxC] = reinterpret_cast<Rec<T>(*)[kMaxC]>(pc_smem);  // [slot][CTA]
  Rec<T>& stage = recv[kSlots][0];                                     // this CTA's candidate, before it is pushed
  Rec<T>& zero = recv[kSlots][1];                                      // stands in for the row of an unusable pivot
  T* mult = reinterpret_cast<T*>(pc_smem + fixed_bytes<T>());          // [column][row]: multipliers
  const int ldm = lds_of<T>(rows_per_cta);
  T(*l11)[NB + 1] = reinterpret_cast<T(*)[NB + 1]>(mult + NB * ldm);  // H = 2: the left half's rows at the diagonal
  T(*u12)[NB + 1] = l11 + NB;                                         // and their entries in the right half
  __shared__ uint64_t bars[kSlots];
  __shared__ Key red_k[2][kW];  // by column parity: a warp may be a column ahead of another's reads
  __shared__ uint32_t red_i[2][kW];
  __shared__ int s_failed;
  __shared__ int s_piv[NB * H];

  const int C = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rbase = k + g * rows_per_cta;
  const int rcount = max(0, min(rows_per_cta, n - rbase));
  const long long limit = min(spin_limit(), 1ll << 22);  // a try_wait may itself suspend for a while

  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&bars[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < kCols<T>) zero.row[tid] = T(0);
  allow_next();
  wait_previous();
  if (tid == 0) s_failed = 0;

  // row r of this thread: local row tid + kThreads * r, its place (the global row it will be written to), the
  // number of its multipliers in this half (all until it is chosen as a pivot; 0 for rows beyond the panel)
  T x[R][NB];
  int place[R], steps[R];
  bool live[R], any[R];  // any: this warp has rows in slot r
  auto load = [&](int base, int hb) {  // the rows' entries in columns [base, base + hb)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int l = tid + kThreads * r;
      const T* src = W + int64_t(rbase + l) * ld + k + base;
      if (l < rcount && hb == NB && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
        for (int c = 0; c < NB; c += kElems) {
          const uint4 w = *reinterpret_cast<const uint4*>(src + c);
          memcpy(&x[r][c], &w, 16);
        }
      } else {
#pragma unroll
        for (int c = 0; c < NB; ++c) x[r][c] = (l < rcount && c < hb) ? src[c] : T(0);
      }
    }
  };
  const int hb0 = H == 1 ? nb : NB;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    any[r] = wid * 32 + kThreads * r < rcount;
    const int l = tid + kThreads * r;
    live[r] = l < rcount;
    place[r] = rbase + l;
    steps[r] = live[r] ? hb0 : 0;
  }
  load(0, hb0);
  cluster_barrier();  // every CTA's barriers are ready (and every row is read) before anyone publishes

  // This thread's candidate for column j (its place, kNoRow if none, and slot) and its warp's, to red_*[j & 1].
  uint32_t own_row = kNoRow;
  int own_slot = 0;
  auto search = [&](int j, Key key, uint32_t row, int slot) {
    own_row = row;
    own_slot = slot;
    warp_best(key, row);
    if (lane == 0) { red_k[j & 1][wid] = key; red_i[j & 1][wid] = row; }
  };
  // Behind a barrier: the CTA's candidate from its warps', published to every CTA by the warp that holds it.
  // Entries x[.][0..) are columns j, j + 1, ...
  auto publish = [&](int j, int hend, auto window) {
    constexpr int WD = decltype(window)::value;
    const int s = j % kSlots;
    Key key = red_k[j & 1][lane & (kW - 1)];
    uint32_t row = red_i[j & 1][lane & (kW - 1)];
    const int words = kHeads + (hend - j + kElems - 1) / kElems;
    if (C > 1 && tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(&bars[s])), "r"(uint32_t(C * 16 * words))
                   : "memory");
    warp_best(key, row);
    const bool won = own_row == row && row != kNoRow, none = row == kNoRow;  // none: a CTA without rows left
    if (!__any_sync(0xffffffffu, won || (none && tid == 0))) return;
    Rec<T>* own = C == 1 ? &recv[s][0] : &stage;
    if (won) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (own_slot == r) {
#pragma unroll
          for (int c = 0; c < WD; c += kElems) {
            uint4 w;
            memcpy(&w, &x[r][c], 16);
            *reinterpret_cast<uint4*>(&own->row[c]) = w;
          }
          own->rinv[0] = T(1) / x[r][0];
        }
    }
    if (won || (none && tid == 0)) own->head = put_head(key, row);
    if (C == 1) return;
    __syncwarp();
    if (lane < words) {
      const uint4 w = reinterpret_cast<const uint4*>(&stage)[lane];
      const uint32_t dst = saddr(&recv[s][g]) + 16 * lane, bar = saddr(&bars[s]);
#pragma unroll 4
      for (int d = 0; d < C; ++d) push16(in_cta(dst, d), w, in_cta(bar, d));
    }
    __syncwarp();
  };

  auto first_column = [&](int j, int hend) {
    Key key = 0;
    uint32_t row = kNoRow;
    int slot = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Key kv = key_of(x[r][0]);
      if (live[r] && (kv > key || (kv == key && uint32_t(place[r]) < row))) { key = kv; row = uint32_t(place[r]); slot = r; }
    }
    search(j, key, row, slot);
    __syncthreads();
    publish(j, hend, Int<NB>{});
  };

  bool failed = false;
  // Columns [base + j0, base + j1) of the half that ends at hend, with the entries x[.][0..WD) still to be eliminated at
  // the first.
  auto steps_of = [&](int base, int hend, int j0, int j1, auto window) {
    constexpr int WD = decltype(window)::value;
    for (int j = base + j0; j < base + j1; ++j) {
      const int s = j % kSlots, diag = k + j;
      int gw = 0;
      if (C == 1) {
        __syncthreads();
      } else {
        const uint32_t bar = saddr(&bars[s]), parity = uint32_t(j / kSlots) & 1u;
        long long it = 0;
        while (!phase_done(bar, parity))
          if (++it > limit) {
            status_error(st, UPDES_ERR_TIMEOUT);
            atomicCAS(&st->timeout_tag, 0, 4);
            s_failed = 1;
            break;
          }
        const uint4 h = recv[s][lane & (C - 1)].head;  // C is a power of two
        Key key;
        get_key(h, key);
        uint32_t row = h.z;
        const uint32_t mine = row;
        warp_best(key, row);
        gw = int(__reduce_min_sync(0xffffffffu, mine == row ? uint32_t(lane & (C - 1)) : 0u + kMaxC)) & (kMaxC - 1);
      }
      const Rec<T>& win = recv[s][gw];
      const uint4 head = win.head;
      Key wkey;
      get_key(head, wkey);
      const uint32_t p = head.z;
      const bool ok = usable(wkey);
      const uint4* pr = reinterpret_cast<const uint4*>(ok ? win.row : zero.row);  // an unusable pivot eliminates nothing
      const T rinv = ok ? win.rinv[0] : T(1);
      T f[kElems];
      auto entries = [&](int c) {  // f = the pivot row's entries c, c + 1, ...
        const uint4 w = pr[c / kElems];
        memcpy(f, &w, 16);
      };
      entries(0);
      T a[R];
      Key key = 0;
      uint32_t row = kNoRow;
      int slot = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (!any[r]) continue;
        if (live[r] && uint32_t(place[r]) == p) {
          live[r] = false;
          place[r] = diag;
          steps[r] = j - base;
        } else if (place[r] == diag && live[r]) {
          place[r] = int(p);
        }
        const T m = x[r][0] * rinv;
        if (live[r]) mult[(j - base) * ldm + tid + kThreads * r] = m;
        a[r] = ok ? -m : T(0);
        x[r][0] = fma_rn(a[r], f[1], x[r][1]);
        const Key kv = key_of(x[r][0]);
        if (live[r] && (kv > key || (kv == key && uint32_t(place[r]) < row))) {
          key = kv;
          row = uint32_t(place[r]);
          slot = r;
        }
      }
      if (j + 1 < hend) search(j + 1, key, row, slot);
      if (any[0]) {
        if constexpr (sizeof(T) == 4) {
#pragma unroll
          for (int c = 0; c < WD; c += kElems) {
            if (c) entries(c);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int i = 0; i < kElems; ++i)
                if (c + i >= 2) x[r][c + i - 1] = fma_rn(a[r], f[i], x[r][c + i]);
          }
        } else {  // the FP64 pipe is what bounds this: a warp's slots without rows are left out
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (any[r]) {
#pragma unroll
              for (int c = 2; c < WD; c += kElems) {
                entries(c);
#pragma unroll
                for (int i = 0; i < kElems; ++i) x[r][c + i - 1] = fma_rn(a[r], f[i], x[r][c + i]);
              }
            }
        }
      }
      __syncthreads();
      if (*static_cast<volatile int*>(&s_failed)) { failed = true; return; }
      if (j + 1 < hend) publish(j + 1, hend, window);
      // off the critical path: the pivot's row of U to its place, the interchange
      if (g == gw && wid == (j % kW))
        for (int c = lane; c < hend - j; c += 32) W[int64_t(diag) * ld + k + j + c] = win.row[c];
      if (tid == 0) {
        s_piv[j] = p == kNoRow ? diag : int(p);
        if (g == 0 && !ok) atomicCAS(&st->lu_info, 0, diag + 1);
      }
    }
  };
  auto eliminate = [&](int base, int hend) {
    const int hb = hend - base;
    constexpr int Q = NB / 4;
    first_column(base, hend);
    steps_of(base, hend, 0, min(hb, Q), Int<NB>{});
    if (!failed) steps_of(base, hend, Q, min(hb, 2 * Q), Int<3 * Q>{});
    if (!failed) steps_of(base, hend, 2 * Q, min(hb, 3 * Q), Int<2 * Q>{});
    if (!failed) steps_of(base, hend, 3 * Q, min(hb, NB), Int<Q>{});
  };
  // Multipliers: the rows' places and counts through shared memory (over the receive slots), a warp per row.
  auto write_back = [&](int base) {
    __syncthreads();
    int2* info = reinterpret_cast<int2*>(pc_smem);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (tid + kThreads * r < rcount) info[tid + kThreads * r] = make_int2(place[r], steps[r]);
    __syncthreads();
    for (int l = wid; l < rcount; l += kW) {
      const int2 q = info[l];
      for (int c = lane; c < q.y; c += 32) W[int64_t(q.x) * ld + k + base + c] = mult[c * ldm + l];
    }
  };
  eliminate(0, hb0);
  int place1[R];  // H = 2: where the left half's multipliers are
  if constexpr (H == 2) {
    // The rows do not move for the right half either: a thread reads its rows' entries where they are.  Every CTA passes
    // every cluster barrier, failed or not.
    if (!failed) {
      write_back(0);
      load(NB, NB);
    }
    cluster_barrier();  // every row of the right half is read, every multiplier is written
    if (!failed) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        place1[r] = place[r];
        steps[r] = live[r] ? NB : 0;
        if (tid + kThreads * r < rcount && !live[r])  // a pivot row of the left half
#pragma unroll
          for (int c = 0; c < NB; ++c) W[int64_t(place[r]) * ld + k + NB + c] = x[r][c];
      }
    }
    cluster_barrier();
    if (!failed) {
      for (int e = tid; e < NB * NB; e += kThreads) {
        const int i = e / NB, c = e % NB;
        l11[i][c] = __ldcg(W + int64_t(k + i) * ld + k + c);
        u12[i][c] = __ldcg(W + int64_t(k + i) * ld + k + NB + c);
      }
      __syncthreads();
      if (wid == 0) {  // u12 by forward substitution, a column per lane (in every CTA: cheaper than handing it round)
        T u[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          T v = u12[i][lane];
#pragma unroll
          for (int j = 0; j < i; ++j) v = fma_rn(-l11[i][j], u[j], v);
          u[i] = v;
          u12[i][lane] = v;
        }
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < NB; ++j) {  // in the order of the elimination
        T m[R];
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = tid + kThreads * r < rcount ? -mult[j * ldm + tid + kThreads * r] : T(0);
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          const T f = u12[j][c];
#pragma unroll
          for (int r = 0; r < R; ++r) x[r][c] = fma_rn(m[r], f, x[r][c]);
        }
      }
    }
    cluster_barrier();  // every CTA has read the right half's rows at the diagonal
    if (!failed) {
      if (g == 0)
        for (int e = tid; e < NB * NB; e += kThreads) W[int64_t(k + e / NB) * ld + k + NB + e % NB] = u12[e / NB][e % NB];
      eliminate(NB, 2 * NB);
    }
    if (!failed) {
      write_back(NB);
      // the left half's multipliers follow the rows that the right half's interchanges moved
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (tid + kThreads * r < rcount && place[r] != place1[r])
#pragma unroll
          for (int c = 0; c < NB; ++c) x[r][c] = __ldcg(W + int64_t(place1[r]) * ld + k + c);
    }
    cluster_barrier();
    if (!failed) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (tid + kThreads * r < rcount && place[r] != place1[r])
#pragma unroll
          for (int c = 0; c < NB; ++c) W[int64_t(place[r]) * ld + k + c] = x[r][c];
    }
  } else if (!failed) {
    write_back(0);
  }
  if (failed) {
    // let stores of the other CTAs that are still on their way land before the shared memory goes away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  } else {
    if (g == 0) {
      if (tid < nb) piv[k + tid] = s_piv[tid];
      if (swap_map && wid == 0) {
        // net permutation of the interchanges: content tracking over <= 2 nb rows
        __shared__ int rows_s[2 * NB * H], cont_s[2 * NB * H];
        for (int i = lane; i < nb; i += 32) rows_s[i] = cont_s[i] = k + i;
        int cnt = nb;
        __syncwarp();
        for (int i = 0; i < nb; ++i) {
          const int p = s_piv[i];
          if (p == k + i) continue;
          int found = -1;
          if (p < k + nb) {
            found = p - k;  // the panel's own rows sit at their place in the list
          } else {
            for (int q = nb + lane; q < cnt; q += 32)
              if (rows_s[q] == p) found = q;
            found = __reduce_max_sync(0xffffffffu, found);
          }
          if (found < 0) {
            if (lane == 0) rows_s[cnt] = cont_s[cnt] = p;
            found = cnt++;
            __syncwarp();
          }
          if (lane == 0) {
            const int a = cont_s[i];
            cont_s[i] = cont_s[found];
            cont_s[found] = a;
          }
          __syncwarp();
        }
        for (int q = lane; q < cnt; q += 32) {
          swap_map[1 + q] = rows_s[q];
          swap_map[129 + q] = cont_s[q];
        }
        if (lane == 0) swap_map[0] = cnt;
      }
    }
  }
  __syncthreads();
  cluster_barrier();
}

template <typename T>
using PanelKernel = void (*)(T*, int64_t, int, int, int, int, int32_t*, int32_t*, DeviceStatus*);
template <typename T>
PanelKernel<T> kernel_of(int rows) {  // rows per thread
  constexpr int NB = kCols<T>;
  return rows <= 1 ? panel_cluster_kernel<T, 1, NB, 1>
                   : rows == 2 ? panel_cluster_kernel<T, 2, NB, 1> : panel_cluster_kernel<T, 3, NB, 1>;
}
PanelKernel<float> halves_kernel_of(int rows) {
  constexpr int NB = kCols<float> / 2;
  return rows <= 4 ? panel_cluster_kernel<float, 4, NB, 2>
                   : rows == 5 ? panel_cluster_kernel<float, 5, NB, 2> : panel_cluster_kernel<float, 6, NB, 2>;
}

// The largest cluster (16, 8 or 0) this device can keep resident with the kernels' largest shared memory; sets the
// kernels' attributes on the way.
template <typename T>
int max_cluster() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (const int v = known[dev].load()) return v - 1;
  int best = 16;
  auto check = [&](const void* kern, size_t smem) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      best = 0;
    while (best) {
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim = {unsigned(best), 1, 1};
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(best);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1) break;
      best = best == 16 ? 8 : 0;
    }
  };
  for (int r = 1; r <= kMaxRows; ++r) check((const void*)kernel_of<T>(r), smem_bytes<T>(kThreads * r, kCols<T>, 1));
  if constexpr (sizeof(T) == 4)
    for (int r = kMaxRows + 1; r <= 2 * kMaxRows; ++r)
      check((const void*)halves_kernel_of(r), smem_bytes<T>(kThreads * r, kCols<T> / 2, 2));
  (void)cudaGetLastError();
  known[dev].store(best + 1);
  return best;
}

// CTAs for a panel of m rows: for floats the fewest that keep one row a thread (64 columns of 3,000 rows: 78 us on 16
// CTAs of one row a thread, 129 on 4 of three); for doubles 64 rows a CTA, because every
// row costs the SM's FP64 pipe (32 columns of 2,000 rows: 71 us at 64 rows a CTA until 16 CTAs are used up, 90 at 256).
template <typename T>
int panel_cluster_ctas(int m, int cmax) {
  constexpr int per = sizeof(T) == 4 ? 256 : 64;
  int C = 1;
  while (C < cmax && m > C * per) C *= 2;
  return C;
}

template <typename T>
int launch(T* W, int64_t ld, int n, int k, int w, int32_t* piv, int32_t* swap_map, DeviceStatus* st, cudaStream_t s,
           bool after_kernel) {
  const int m = n - k;
  const int cmax = max_cluster<T>();
  if (cmax == 0 || w > kCols<T> || m < w) return UPDES_ERR_UNSUPPORTED;
  const int C = panel_cluster_ctas<T>(m, cmax);
  const int rows = int(ceil_div(m, C)), per_thread = int(ceil_div(rows, kThreads));
  // In halves only where whole rows do not fit the registers: at 12,000 rows 130 us against 118, at 6,000 104 against 92
  const bool halves = sizeof(T) == 4 && w == kCols<T> && per_thread > kMaxRows;
  if (per_thread > (halves ? 2 : 1) * kMaxRows) return UPDES_ERR_UNSUPPORTED;
  PanelKernel<T> kern = kernel_of<T>(per_thread);
  if constexpr (sizeof(T) == 4)
    if (halves) kern = halves_kernel_of(per_thread);
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {unsigned(C), 1, 1};
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_next
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes<T>(rows, halves ? kCols<T> / 2 : kCols<T>, halves ? 2 : 1);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = after_kernel ? 2 : 1;
  StatScope sc(kStatPanel, s, double(m) * w * w, double(m) * w * 2.0 * sizeof(T));
  UPDES_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, W, ld, n, k, w, rows, piv, swap_map, st));
  stats_count_launch(1);
  return UPDES_OK;
}

}  // namespace

int panel_cluster(float* W, int64_t ld, int n, int k, int w, int32_t* piv, int32_t* swap_map, DeviceStatus* st,
                  cudaStream_t s, bool after_kernel) {
  return launch<float>(W, ld, n, k, w, piv, swap_map, st, s, after_kernel);
}

int panel_cluster(double* W, int64_t ld, int n, int k, int w, int32_t* piv, int32_t* swap_map, DeviceStatus* st,
                  cudaStream_t s, bool after_kernel) {
  return launch<double>(W, ld, n, k, w, piv, swap_map, st, s, after_kernel);
}
