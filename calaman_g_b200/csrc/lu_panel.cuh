// lu_panel.cuh -- the panel factorisation of the blocked LU with partial
// pivoting, one thread-block cluster per panel, one panel row per thread.
#pragma once

#include <cooperative_groups.h>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace clm {

template <typename T> __device__ __forceinline__ double safe_min();
template <> __device__ __forceinline__ double safe_min<float>() { return FLT_MIN; }
template <> __device__ __forceinline__ double safe_min<double>() { return DBL_MIN; }
template <> __device__ __forceinline__ double safe_min<float2>() { return FLT_MIN; }
template <> __device__ __forceinline__ double safe_min<double2>() { return DBL_MIN; }

template <typename T> __device__ __forceinline__ T shfl(T v, int src);
template <> __device__ __forceinline__ float shfl<float>(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <> __device__ __forceinline__ double shfl<double>(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <> __device__ __forceinline__ float2 shfl<float2>(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
template <> __device__ __forceinline__ double2 shfl<double2>(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// A pivot candidate: the IEEE-754 bits of |Re| + |Im| plus one (bits order
// non-negative values as the values themselves), 0 for NaN, and the row's
// current position. Float rows need 32 bits of key, the others 64. A thread
// without a candidate carries key 0 at position INT_MAX, so that a NaN row
// still wins over it: a column of NaNs yields its first row, as IxAMAX does.
struct PivotCand {
  unsigned hi, lo;
  int pos;
};
template <typename T>
__device__ __forceinline__ PivotCand pivot_cand(T x, int pos, bool live) {
  PivotCand c{0u, 0u, INT_MAX};
  if (live) {
    c.pos = pos;
    if constexpr (std::is_same<T, float>::value) {
      const float v = fabsf(x);
      if (v >= 0.f) c.hi = __float_as_uint(v) + 1u;
    } else {
      const double v = abs1(x);
      if (v >= 0.0) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v) + 1ull;
        c.hi = (unsigned)(b >> 32);
        c.lo = (unsigned)b;
      }
    }
  }
  return c;
}
// The largest key of the warp, the smallest position among its holders.
template <typename T>
__device__ __forceinline__ PivotCand warp_best(PivotCand c) {
  const unsigned full = 0xffffffffu;
  PivotCand m;
  m.hi = __reduce_max_sync(full, c.hi);
  bool win = c.hi == m.hi;
  m.lo = 0u;
  if constexpr (!std::is_same<T, float>::value) {
    m.lo = __reduce_max_sync(full, win ? c.lo : 0u);
    win = win && c.lo == m.lo;
  }
  m.pos = (int)__reduce_min_sync(full, win ? (unsigned)c.pos : (unsigned)INT_MAX);
  return m;
}

__device__ __forceinline__ unsigned cluster_addr(const void *p, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(tc::saddr(p)), "r"(rank));
  return r;
}
// 16 bytes into another CTA's shared memory, counted on its mbarrier.
__device__ __forceinline__ void st_async16(unsigned dst, uint4 v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(dst),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}

// How the rows below a pivot are scaled (xGETF2): by its reciprocal, by
// division where the reciprocal could overflow, not at all for a zero pivot or
// a column of NaNs.
enum PivotScale { kScaleReciprocal = 0, kScaleDivide = 1, kScaleNone = 2 };

// What a CTA publishes for one pivot column: its candidate, how to scale by
// the candidate's pivot element and its reciprocal, and the candidate's row.
template <typename T, int KB>
struct alignas(16) PivotSlot {
  unsigned hi, lo;
  int pos, scale;
  alignas(16) T rcp[16 / sizeof(T)];
  alignas(16) T row[KB];
};

constexpr int kPanelMaxCluster = 8;

constexpr unsigned kGaveUp = 0xffffffffu;  // above the key of every candidate
constexpr long long kPanelDrainTries = 1ll << 12;  // for pushes under way when a panel is given up

// Bytes of dynamic shared memory the kernel below takes with nt threads.
template <typename T, int KB>
inline std::size_t panel_rows_smem(int nt) { return sizeof(T) * (std::size_t)KB * nt; }

// The h x kb panel (h = n - k) of A, factored in place with partial pivoting
// (largest |Re| + |Im|, first position on ties). Thread (rank, tid) keeps row
// rank * blockDim + tid of the panel for the whole kernel, so the panel is read
// and written once and a pivot column is a chain of: warp and CTA argmax (one
// CTA barrier), the CTA's winner pushed with its row into every CTA's slot
// (16-byte st.async, counted on that CTA's mbarrier), the argmax over the <= 8
// slots, the row update. Rows never move between threads: a row carries its
// position, and a pivot exchange swaps two positions.
//
// Register place i holds column j + i at step j: the update writes one place
// down, so one rolled body with static register indices serves every column
// (unrolled by eight columns its instruction fetch cost more than the chain).
// Multipliers leave for shared memory as they are formed; a pivot row stops
// moving and keeps its part of U in its registers.
//
// Slots and mbarriers alternate by column: a CTA's push for column j + 2 needs
// every CTA's push for column j + 1, which each CTA issues after a barrier
// behind its last read of column j.
//
// Bound: the latency of that chain, once per column. Waits are bounded. A warp
// whose wait runs out uses nothing of the slots; in the place of its candidate for
// the next column it leaves a key above all others, at which its whole CTA leaves
// the loop, and it raises a flag in every CTA, read behind the cluster barrier at
// the end. Permutation and map are written only if no CTA gave up. Otherwise the
// panel's rows are in no defined order, its pivots and its map are the identity
// (what runs behind it stays in range), info = n + 1, and every CTA waits once
// more, bounded, for pushes under way to it.
template <typename T, int KB, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    lu_panel_rows_kernel(int n, T *__restrict__ A, int lda, int k, int kb, int *__restrict__ ipiv,
                         int *__restrict__ perm, int *__restrict__ g_map_pos, int *__restrict__ g_map_src,
                         int *__restrict__ g_map_count, int *__restrict__ info, const PanelWait wait) {
  namespace cgr = cooperative_groups;
  constexpr int U = 8;                    // places per guarded group of the update
  constexpr int V = 16 / (int)sizeof(T);  // elements per 16-byte piece
  constexpr int kHead = 2;                // 16-byte pieces before the row of a slot
  using Slot = PivotSlot<T, KB>;
  static_assert(sizeof(Slot) == 16 * kHead + sizeof(T) * KB && KB % U == 0, "slot layout");
  cgr::cluster_group cluster = cgr::this_cluster();
  const int rank = (int)cluster.block_rank(), ncta = (int)cluster.num_blocks();
  const int lg = 31 - __clz(ncta);  // the cluster's size is a power of two
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
  const int h = n - k;
  const int gi = rank * nt + tid;
  const bool has = gi < h;
  T *P = A + (std::size_t)k * lda + k;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *mult = reinterpret_cast<T *>(smem_raw) + tid;  // this row's multipliers, nt apart
  __shared__ Slot slot[2][kPanelMaxCluster];
  __shared__ Slot stage;
  __shared__ unsigned wkey[2][2][MAXT / 32];
  __shared__ int wpos[2][MAXT / 32];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ int below[2];
  __shared__ int failed;  // a warp of any CTA gave up

  if (tid == 0) {
    failed = 0;
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  T r[KB];
#pragma unroll
  for (int c = 0; c < KB; ++c) r[c] = (has && c < kb) ? P[(std::size_t)c * lda + gi] : elem<T>::zero();
  if (ncta > 1) cluster.sync();  // the mbarriers and the flag exist before any push

  bool active = has;
  int pos = gi, own = kb, first_zero = -1;  // own: the step at which this row became the pivot
  auto warp_candidate = [&](int buf) {
    const PivotCand c = warp_best<T>(pivot_cand<T>(r[0], pos, active));
    if (lane == 0) {
      wkey[buf][0][warp] = c.hi;
      if constexpr (!std::is_same<T, float>::value) wkey[buf][1][warp] = c.lo;
      wpos[buf][warp] = c.pos;
    }
  };
  warp_candidate(0);
  int j = 0;
#pragma unroll 1
  for (; j < kb; ++j) {
    const int par = j & 1;
    const int live = KB - j;                          // places that hold columns of the panel
    const int pieces = (live + U - 1) / U * (U / V);  // 16-byte pieces of the row that still matter
    // ---- this CTA's candidate, from its warps' ----
    if (ncta > 1 && tid == 0) tc::mbar_expect_tx(&bar[par], (unsigned)((kHead + pieces) * 16) << lg);
    __syncthreads();
    PivotCand c;
    c.hi = lane < nwarps ? wkey[par][0][lane] : 0u;
    c.lo = 0u;
    if constexpr (!std::is_same<T, float>::value) c.lo = lane < nwarps ? wkey[par][1][lane] : 0u;
    c.pos = lane < nwarps ? wpos[par][lane] : INT_MAX;
    c = warp_best<T>(c);
    if (ncta > 1 && c.hi == kGaveUp) break;
    const bool mine = active && pos == c.pos;
    // the winner's warp publishes it; a CTA without candidates publishes that
    if (__any_sync(0xffffffffu, mine) || (c.pos == INT_MAX && warp == 0)) {
      if (mine || (c.pos == INT_MAX && lane == 0)) {
        Slot *const out = ncta > 1 ? &stage : &slot[par][0];
        out->hi = c.hi;
        out->lo = c.lo;
        out->pos = c.pos;
        const bool zero = (c.hi == 0u && c.lo == 0u) || is_zero(r[0]);
        out->scale = zero ? kScaleNone : abs1(r[0]) >= safe_min<T>() ? kScaleReciprocal : kScaleDivide;
#pragma unroll
        for (int i = 0; i < KB; i += V) {
          union {
            T e[V];
            uint4 q;
          } w;
#pragma unroll
          for (int e = 0; e < V; ++e) w.e[e] = r[i + e];
          *reinterpret_cast<uint4 *>(&out->row[i]) = w.q;
        }
        out->rcp[0] = zero ? elem<T>::one() : divide(elem<T>::one(), r[0]);
      }
      if (ncta > 1 && (j < wait.drop_from || rank + 1 < ncta)) {
        __syncwarp();
        for (int t = lane; t < (kHead + pieces) << lg; t += 32) {
          const int q = t & (ncta - 1), at = t >> lg;
          st_async16(cluster_addr(reinterpret_cast<uint4 *>(&slot[par][rank]) + at, q),
                     reinterpret_cast<const uint4 *>(&stage)[at], cluster_addr(&bar[par], q));
        }
      }
    }
    int from = 0;
    if (ncta > 1) {
      bool arrived = false;
      for (int i = 0; i < wait.tries && !arrived; ++i) arrived = tc::mbar_try_wait(&bar[par], (unsigned)(j >> 1) & 1u);
      c.hi = lane < ncta ? slot[par][lane].hi : 0u;
      c.lo = lane < ncta ? slot[par][lane].lo : 0u;
      const int p = lane < ncta ? slot[par][lane].pos : INT_MAX;
      c.pos = p;
      const bool all = __all_sync(0xffffffffu, arrived);
      c = warp_best<T>(c);
      if (!all) {  // the slots say nothing
        if (lane == 0) wkey[par ^ 1][0][warp] = kGaveUp;
        if (lane < ncta) *cluster.map_shared_rank(&failed, lane) = 1;
        continue;
      }
      from = __ffs(__ballot_sync(0xffffffffu, p == c.pos)) - 1;
    } else {
      __syncthreads();
    }
    // ---- swap positions, scale by the pivot; the next column's element first,
    // so that its candidate is under way during the rest of the update ----
    const Slot &win = slot[par][from];
    const int how = win.scale;
    if (how == kScaleNone && first_zero < 0) first_zero = j;
    if (rank == 0 && tid == 0) ipiv[k + j] = k + c.pos;
    T l = elem<T>::zero();
    if (active) {
      if (pos == c.pos) {
        active = false;
        pos = own = j;
      } else {
        if (pos == j) pos = c.pos;
        l = how == kScaleReciprocal ? mul(r[0], win.rcp[0]) : how == kScaleDivide ? divide(r[0], win.row[0]) : r[0];
        mult[j * nt] = l;
        r[0] = sub(r[1], mul(l, win.row[1]));
      }
    }
    warp_candidate(par ^ 1);
    if (active) {
      auto update = [&](auto places) {
#pragma unroll
        for (int i = 0; i < places; i += V) {
          union {
            T e[V];
            uint4 q;
          } w;
          w.q = *reinterpret_cast<const uint4 *>(&win.row[i]);
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (i + e > 1) r[i + e - 1] = sub(r[i + e], mul(l, w.e[e]));
        }
      };
      // two unguarded lengths: guards between pieces kept each piece's load
      // behind the piece before it (float32, 32 columns: 490 cycles a column)
      if (live > KB / 2) update(std::integral_constant<int, KB>{});
      else update(std::integral_constant<int, KB / 2>{});
    }
  }

  // ---- rows back at their positions; what moved, for the swaps elsewhere ----
  if (has) {
    T *row = P + pos;
#pragma unroll 4
    for (int c = 0; c < own; ++c) row[(std::size_t)c * lda] = mult[c * nt];
    row += (std::size_t)own * lda;
#pragma unroll
    for (int c = 0; c < KB; ++c)
      if (own + c < kb) row[(std::size_t)c * lda] = r[c];
  }
  const bool moved = has && (pos < kb || pos != gi);
  const int old = moved ? perm[k + gi] : 0;
  // rows below the top kb only ever receive rows of the top kb (the first
  // threads of rank 0), which are appended to the map behind the top rows
  const bool down = has && gi < kb && pos >= kb;
  const unsigned downs = __ballot_sync(0xffffffffu, down);
  if (rank == 0 && warp < 2 && lane == 0) below[warp] = __popc(downs);
  if (ncta > 1) cluster.sync();  // every read of perm is done, every flag is there
  else __syncthreads();
  if (failed) {
    if (rank == 0 && tid < kb) {  // at least 64 threads
      ipiv[k + tid] = k + tid;
      g_map_pos[tid] = g_map_src[tid] = k + tid;
      if (tid == 0) {
        *g_map_count = kb;
        info[0] = n + 1;
      }
    }
    // the column given up and the one behind it, which a peer may have entered
    if (ncta > 1 && tid == 0)
      for (int c = j - 1; c <= j; ++c) tc::mbar_wait(&bar[c & 1], (unsigned)(c >> 1) & 1u, kPanelDrainTries);
    return;
  }
  if (moved) perm[k + pos] = old;
  if (has && pos < kb) {
    g_map_pos[pos] = k + pos;
    g_map_src[pos] = k + gi;
  }
  if (down) {
    const int e = kb + (warp == 1 ? below[0] : 0) + __popc(downs & ((1u << lane) - 1u));
    g_map_pos[e] = k + pos;
    g_map_src[e] = k + gi;
  }
  if (rank == 0 && tid == 0) {
    *g_map_count = kb + below[0] + (nwarps > 1 ? below[1] : 0);
    if (first_zero >= 0 && info[0] == 0) info[0] = k + first_zero + 1;
  }
}

}  // namespace clm
