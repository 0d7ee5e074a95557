// lu.cu -- LU with partial pivoting (xGETRF semantics) and the n-right-hand-
// side solve (xGETRS, no transpose) for the Pade denominator q_m(A), written
// for sm_100a without cuSOLVER (the reference reaches cuSOLVER through
// WarpWraps: src/expm/pade.cppm:186-188).
//
// Blocked right-looking factorisation, panel width kb <= 64:
//   1. panel: heights up to 4096 in lu_panel.cuh (one row per thread, a cluster
//      of eight CTAs); taller ones in lu_panel_kernel below, whose cluster
//      (<= 8 CTAs) holds the h x kb panel in the CTAs' shared memory. Per pivot
//      column there:
//        - every CTA reduces its local pivot candidate (largest |Re|+|Im|,
//          first index on ties -- LAPACK IxAMAX) and publishes it, with the
//          candidate's whole row, into a double-buffered slot;
//        - ONE cluster barrier;
//        - every CTA fetches all candidates and their rows (and row j) over
//          distributed shared memory in a single round trip, and agrees on
//          the pivot without further communication;
//        - one fused pass swaps, scales by the pivot's reciprocal (as xGETF2
//          does above the safe minimum), applies the rank-1 update to its own
//          rows and already forms the NEXT column's local candidate.
//      That is two CTA barriers and one cluster barrier per column.
//   2. swap + TRSM: one warp per column outside the panel applies the panel's
//      row permutation (a compact gather of <= 2 kb rows) and, right of the
//      panel and in a right-hand side, solves with the unit-lower L11 held in
//      shared memory.
//   3. trailing update: A22 -= L21 U12 on the tensor-core GEMM.
// getrf_solve runs the forward substitution of its right-hand side beside the
// factorisation, then blocked backward substitution (diagonal blocks per warp,
// off-diagonal blocks on the GEMM); getrs gathers the right-hand side through
// the accumulated row permutation and runs both.
#include <cooperative_groups.h>
#include <climits>
#include <type_traits>

#include "kernels.cuh"
#include "lu_panel.cuh"

namespace cg = cooperative_groups;

namespace clm {

namespace {

constexpr int kMaxKb = 64;
constexpr int kPanelThreads = 512;
constexpr int kMaxCluster = 8;
constexpr std::size_t kPanelSmemBudget = 176 * 1024;  // bytes of panel per CTA

// scratch: ipiv[n] | perm[n] | two row maps (of even and of odd panels: a
// panel's swaps are still replayed while the next panel writes its own), each
// map_pos[2*kMaxKb] | map_src[2*kMaxKb] | map_count
struct RowMap {
  int *pos, *src, *count;
};
struct LuScratch {
  int *ipiv, *perm;
  RowMap map[2];
};
inline LuScratch carve_lu(void *base, int n) {
  Layout L(base);
  LuScratch s;
  s.ipiv = L.take<int>(n);
  s.perm = L.take<int>(n);
  for (RowMap &m : s.map) {
    m.pos = L.take<int>(2 * kMaxKb);
    m.src = L.take<int>(2 * kMaxKb);
    m.count = L.take<int>(1);
  }
  return s;
}

__host__ __device__ inline std::size_t align16(std::size_t x) { return (x + 15) & ~std::size_t(15); }

// Offsets of the panel kernel's shared-memory regions (host and device agree).
struct PanelSmem {
  std::size_t S, slot_row, slot_diag, cand, oldrow, slot_val, slot_idx, cand_val, cand_idx, red_val, red_idx, plist, flags, map_pos, map_org, total;
};
template <typename T>
__host__ __device__ inline PanelSmem panel_smem(int rpc, int kb) {
  PanelSmem o;
  std::size_t at = 0;
  o.S = at; at = align16(at + sizeof(T) * (std::size_t)rpc * kb);
  o.slot_row = at; at = align16(at + sizeof(T) * 2 * kb);
  o.slot_diag = at; at = align16(at + sizeof(T) * 2 * kb);
  o.cand = at; at = align16(at + sizeof(T) * kMaxCluster * kb);
  o.oldrow = at; at = align16(at + sizeof(T) * kb);
  o.slot_val = at; at = align16(at + sizeof(double) * 2);
  o.slot_idx = at; at = align16(at + sizeof(int) * 2);
  o.cand_val = at; at = align16(at + sizeof(double) * kMaxCluster);
  o.cand_idx = at; at = align16(at + sizeof(int) * kMaxCluster);
  o.red_val = at; at = align16(at + sizeof(double) * (kPanelThreads / 32));
  o.red_idx = at; at = align16(at + sizeof(int) * (kPanelThreads / 32));
  o.plist = at; at = align16(at + sizeof(int) * kb);
  o.flags = at; at = align16(at + sizeof(int) * 4);
  o.map_pos = at; at = align16(at + sizeof(int) * 2 * kb);
  o.map_org = at; at = align16(at + sizeof(int) * 2 * kb);
  o.total = at;
  return o;
}

// (value, index) max with the first index winning ties
__device__ __forceinline__ void argmax_merge(double &v, int &i, double ov, int oi) {
  if (ov > v || (ov == v && oi < i)) {
    v = ov;
    i = oi;
  }
}

// one element global -> shared, asynchronously (4, 8 or 16 bytes)
template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (sizeof(T) == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
  } else if constexpr (sizeof(T) == 8) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
  }
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::);
}

__device__ __noinline__ void panel_finish(cg::cluster_group &cluster, int rank, int k, int kb,
                                          const int *plist, const int *flags, int *mpos, int *morg,
                                          int *__restrict__ ipiv, int *__restrict__ perm,
                                          int *__restrict__ g_map_pos, int *__restrict__ g_map_src,
                                          int *__restrict__ g_map_count, int *__restrict__ info);

template <typename T>
__global__ void __launch_bounds__(kPanelThreads)
    lu_panel_kernel(int n, T *__restrict__ A, int lda, int k, int kb, int rpc, int *__restrict__ ipiv,
                    int *__restrict__ perm, int *__restrict__ g_map_pos, int *__restrict__ g_map_src,
                    int *__restrict__ g_map_count, int *__restrict__ info) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int ncta = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = blockDim.x;  // a multiple of 32, at most kPanelThreads
  const int h = n - k;
  const int r0 = rank * rpc;
  int rows_here = h - r0;
  rows_here = rows_here < 0 ? 0 : (rows_here > rpc ? rpc : rows_here);

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelSmem o = panel_smem<T>(rpc, kb);
  T *S = reinterpret_cast<T *>(smem_raw + o.S);
  T *slot_row = reinterpret_cast<T *>(smem_raw + o.slot_row);
  T *slot_diag = reinterpret_cast<T *>(smem_raw + o.slot_diag);
  T *cand = reinterpret_cast<T *>(smem_raw + o.cand);
  T *oldrow = reinterpret_cast<T *>(smem_raw + o.oldrow);
  double *slot_val = reinterpret_cast<double *>(smem_raw + o.slot_val);
  int *slot_idx = reinterpret_cast<int *>(smem_raw + o.slot_idx);
  double *cand_val = reinterpret_cast<double *>(smem_raw + o.cand_val);
  int *cand_idx = reinterpret_cast<int *>(smem_raw + o.cand_idx);
  double *red_val = reinterpret_cast<double *>(smem_raw + o.red_val);
  int *red_idx = reinterpret_cast<int *>(smem_raw + o.red_idx);
  int *plist = reinterpret_cast<int *>(smem_raw + o.plist);
  int *flags = reinterpret_cast<int *>(smem_raw + o.flags);  // [0] first zero pivot

  // Work split of the fused pass: ncph adjacent lanes share a row, each taking
  // every ncph-th column, so a row's readers of column j sit in one warp and a
  // __syncwarp orders them before column j is overwritten.
  int ncph = 1;
  while (ncph * 2 <= 32 && ncph * 2 * rpc <= nt) ncph *= 2;
  const int RT = nt / ncph;  // rows covered per sweep
  const int my_c = tid % ncph, my_r = tid / ncph;
  const int iters = (rpc + RT - 1) / RT;  // uniform across the CTA

  // ---- stage the panel rows this CTA owns (all copies in flight at once) ----
  for (int idx = tid; idx < rows_here * kb; idx += nt) {
    const int li = idx % rows_here, c = idx / rows_here;
    cp_async_elem(&S[(std::size_t)c * rpc + li], &A[(std::size_t)(k + c) * lda + (k + r0 + li)]);
  }
  cp_async_wait_all();
  if (tid == 0) flags[0] = -1;
  __syncthreads();

  // local candidate for column 0 (the lane whose phase owns column 0)
  double bv = -1.0;
  int bi = INT_MAX;
  if (my_c == 0)
    for (int li = my_r; li < rows_here; li += RT) argmax_merge(bv, bi, abs1(S[li]), r0 + li);

  for (int j = 0; j < kb; ++j) {
    const int par = j & 1;
    const int owner_j = j / rpc;
    // ---- (1) CTA-wide candidate, published with its row ----
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, bv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      argmax_merge(bv, bi, ov, oi);
    }
    if (lane == 0) {
      red_val[warp] = bv;
      red_idx[warp] = bi;
    }
    __syncthreads();
    if (warp == 0) {
      double v = lane < nt / 32 ? red_val[lane] : -1.0;
      int i = lane < nt / 32 ? red_idx[lane] : INT_MAX;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, off);
        const int oi = __shfl_xor_sync(0xffffffffu, i, off);
        argmax_merge(v, i, ov, oi);
      }
      if (lane == 0) {
        slot_val[par] = v;
        slot_idx[par] = i;
      }
      for (int c = lane; c < kb; c += 32) {
        if (i != INT_MAX) slot_row[par * kb + c] = S[(std::size_t)c * rpc + (i - r0)];
        if (rank == owner_j) slot_diag[par * kb + c] = S[(std::size_t)c * rpc + (j - r0)];
      }
    }
    cluster.sync();

    // ---- (2) one DSMEM round trip: every candidate, its row, and row j ----
    for (int t = tid; t < ncta * kb + kb + ncta; t += nt) {
      if (t < ncta * kb) {
        const int q = t / kb, c = t % kb;
        cand[q * kb + c] = cluster.map_shared_rank(slot_row, q)[par * kb + c];
      } else if (t < ncta * kb + kb) {
        const int c = t - ncta * kb;
        oldrow[c] = cluster.map_shared_rank(slot_diag, owner_j)[par * kb + c];
      } else {
        const int q = t - ncta * kb - kb;
        cand_val[q] = cluster.map_shared_rank(slot_val, q)[par];
        cand_idx[q] = cluster.map_shared_rank(slot_idx, q)[par];
      }
    }
    __syncthreads();

    // ---- (3) the pivot, agreed by every warp from the same data ----
    double pv = lane < ncta ? cand_val[lane] : -1.0;
    int p = lane < ncta ? cand_idx[lane] : INT_MAX;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {  // full butterfly: every lane ends with the winner
      const double ov = __shfl_xor_sync(0xffffffffu, pv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, p, off);
      argmax_merge(pv, p, ov, oi);
    }
    if (p == INT_MAX || p < j) {  // no comparable candidate (NaN column): keep row j
      p = j;
      pv = 0.0;
    }
    const T *pivrow = (p == j) ? oldrow : cand + (p / rpc) * kb;
    const T piv = pivrow[j];
    const bool singular = is_zero(piv);
    const bool use_recip = abs1(piv) >= safe_min<T>();
    const T rpiv = (use_recip && !singular) ? divide(elem<T>::one(), piv) : elem<T>::one();
    auto scale_by_pivot = [&](T x) -> T {
      return singular ? x : (use_recip ? mul(x, rpiv) : divide(x, piv));
    };
    if (tid == 0) {
      plist[j] = p;
      if (pv == 0.0 && flags[0] < 0) flags[0] = j;
    }

    // ---- (4a) the two rows that move, one element per thread: position j
    //      receives the pivot row, position p the old row j (updated) ----
    bv = -1.0;
    bi = INT_MAX;
    const int nextc = j + 1;
    const bool own_j = rank == owner_j;
    const bool own_p = p != j && rank == p / rpc;
    for (int t = tid; t < 2 * kb; t += nt) {
      if (t < kb) {
        if (own_j) S[(std::size_t)t * rpc + (j - r0)] = pivrow[t];
      } else if (own_p) {
        const int c = t - kb;
        const T lp = scale_by_pivot(oldrow[j]);
        T v;
        if (c < j) v = oldrow[c];
        else if (c == j) v = lp;
        else v = sub(oldrow[c], mul(lp, pivrow[c]));
        S[(std::size_t)c * rpc + (p - r0)] = v;
        if (c == nextc) argmax_merge(bv, bi, abs1(v), p);
      }
    }

    // ---- (4b) every other row below j: scale, rank-1 update, next candidate ----
    for (int it = 0; it < iters; ++it) {
      const int li = my_r + it * RT;
      const int gi = r0 + li;
      const bool row_ok = li < rows_here && gi > j && gi != p;
      T xj = elem<T>::zero();
      if (row_ok) xj = S[(std::size_t)j * rpc + li];
      __syncwarp();  // every lane of this row has read column j
      if (!row_ok) continue;
      T *row = S + li;
      const T l = scale_by_pivot(xj);
      // first column >= j in this lane's phase (ncph is a power of two)
      int c = j + ((my_c - j) & (ncph - 1));
      if (c == j) {
        row[(std::size_t)j * rpc] = l;
        c += ncph;
      }
      // four columns at a time, all loads issued before the stores
      for (; c < kb; c += 4 * ncph) {
        T x[4], pr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int cc = c + u * ncph;
          if (cc < kb) {
            x[u] = row[(std::size_t)cc * rpc];
            pr[u] = pivrow[cc];
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int cc = c + u * ncph;
          if (cc < kb) row[(std::size_t)cc * rpc] = sub(x[u], mul(l, pr[u]));
        }
      }
      // this lane's share of the next column's candidate
      if (nextc < kb && ((nextc - my_c) & (ncph - 1)) == 0)
        argmax_merge(bv, bi, abs1(row[(std::size_t)nextc * rpc]), gi);
    }
  }

  // ---- write the factored panel back ----
  __syncthreads();
  for (int idx = tid; idx < rows_here * kb; idx += nt) {
    const int li = idx % rows_here, c = idx / rows_here;
    A[(std::size_t)(k + c) * lda + (k + r0 + li)] = S[(std::size_t)c * rpc + li];
  }

  panel_finish(cluster, rank, k, kb, plist, flags, reinterpret_cast<int *>(smem_raw + o.map_pos),
               reinterpret_cast<int *>(smem_raw + o.map_org), ipiv, perm, g_map_pos, g_map_src,
               g_map_count, info);
}

// Epilogue of the panel kernel: the pivot vector, LAPACK's info, the
// compact row map the swap kernel replays, and the accumulated permutation.
// Ends with the cluster barrier that keeps every CTA's shared memory alive
// until the last remote read of it has completed.
__device__ __noinline__ void panel_finish(cg::cluster_group &cluster, int rank, int k, int kb,
                                          const int *plist, const int *flags, int *mpos, int *morg,
                                          int *__restrict__ ipiv, int *__restrict__ perm,
                                          int *__restrict__ g_map_pos, int *__restrict__ g_map_src,
                                          int *__restrict__ g_map_count, int *__restrict__ info) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (rank != 0) {
    cluster.sync();
    return;
  }
  if (tid < kb) ipiv[k + tid] = k + plist[tid];
  if (tid == 0 && flags[0] >= 0 && info[0] == 0) info[0] = k + flags[0] + 1;

  // ---- compact row map of the panel's swaps (warp 0 of rank 0) ----
  // entries 0..kb-1 are rows k..k+kb-1 in order; extra rows the swaps reached
  // are appended. After replaying the swaps, row pos[e] holds old row org[e].
  if (warp == 0) {
    for (int e = lane; e < kb; e += 32) {
      mpos[e] = k + e;
      morg[e] = k + e;
    }
    __syncwarp();
    int count = kb;
    for (int j = 0; j < kb; ++j) {
      const int b = plist[j];
      int bidx;
      if (b < kb) {
        bidx = b;
      } else {
        bidx = -1;
        for (int base = kb; base < count; base += 32) {
          const int e = base + lane;
          const unsigned hit = __ballot_sync(0xffffffffu, e < count && mpos[e] == k + b);
          if (hit) {
            bidx = base + __ffs(hit) - 1;
            break;
          }
        }
        if (bidx < 0) {
          bidx = count;
          if (lane == 0) {
            mpos[count] = k + b;
            morg[count] = k + b;
          }
          ++count;
        }
      }
      __syncwarp();
      if (lane == 0 && bidx != j) {
        const int t = morg[j];
        morg[j] = morg[bidx];
        morg[bidx] = t;
      }
      __syncwarp();
    }
    int pv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = lane + 32 * q;
      if (e < count) {
        g_map_pos[e] = mpos[e];
        g_map_src[e] = morg[e];
        pv[q] = perm[morg[e]];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = lane + 32 * q;
      if (e < count) perm[mpos[e]] = pv[q];
    }
    if (lane == 0) *g_map_count = count;
  }
  cluster.sync();
}

// Load the kb x kb diagonal block A[k:k+kb, k:k+kb] into shared memory (D[l kb + i]
// = A(k + i, k + l)): a warp per column, 16-byte copies when every column of
// the block starts 16-byte aligned, else one element per copy. (The per-element
// form with an index division per element set the time of the 128-row float32
// solve blocks: 16k copies per CTA.)
template <typename T>
__device__ __forceinline__ void load_diag_block(T *D, const T *A, int lda, int k, int kb) {
  constexpr int V = 16 / sizeof(T);  // elements per 16-byte copy
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const T *base = A + (std::size_t)k * lda + k;
  if (V > 1 && kb % V == 0 && lda % V == 0 && (reinterpret_cast<std::uintptr_t>(base) & 15) == 0) {
    for (int l = threadIdx.x >> 5; l < kb; l += warps)
      for (int i = lane * V; i < kb; i += 32 * V) {
        const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(&D[l * kb + i]));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(&base[(std::size_t)l * lda + i]));
      }
  } else {
    for (int l = threadIdx.x >> 5; l < kb; l += warps)
      for (int i = lane; i < kb; i += 32) cp_async_elem(&D[l * kb + i], &base[(std::size_t)l * lda + i]);
  }
  cp_async_wait_all();
}

// ---- swap + TRSM of one panel for columns outside it: one warp per column ----
// Columns [c0, c0 + nright) right of the panel, then nrhs columns of a right-
// hand side B (both: swaps, then the solve with the unit-lower L11), then the
// nleft first columns of A (swaps only). The solved rows of a right-hand side
// go to rows k .. k + kb - 1 of X; the rows the swaps moved down stay in B,
// whose rows below the panel are still being updated.
template <typename T>
__global__ void __launch_bounds__(256)
    lu_swap_trsm_kernel(T *__restrict__ A, int lda, int k, int kb, int c0, int nright, int nleft,
                        T *__restrict__ B, int ldb, T *__restrict__ X, int ldx, int nrhs,
                        const int *__restrict__ map_pos, const int *__restrict__ map_src,
                        const int *__restrict__ map_count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *L = reinterpret_cast<T *>(smem_raw);  // kb x kb, column-major
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int ci = blockIdx.x * warps + (threadIdx.x >> 5);
  if ((int)blockIdx.x * warps < nright + nrhs) load_diag_block(L, A, lda, k, kb);  // holds a column to solve
  __syncthreads();
  if (ci >= nright + nrhs + nleft) return;
  const bool rhs = ci >= nright && ci < nright + nrhs, left = ci >= nright + nrhs;
  T *col = rhs ? B + (std::size_t)(ci - nright) * ldb : A + (std::size_t)(left ? ci - nright - nrhs : c0 + ci) * lda;
  const int cnt = *map_count;
  T v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = lane + 32 * q;
    v[q] = e < cnt ? col[map_src[e]] : elem<T>::zero();
  }
  __syncwarp();
  if (left) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = lane + 32 * q;
      if (e < cnt) col[map_pos[e]] = v[q];
    }
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = lane + 32 * q;
    if (e >= kb && e < cnt) col[map_pos[e]] = v[q];
  }
  T x0 = v[0], x1 = v[1];  // rows k+lane, k+lane+32
  for (int l = 0; l < kb; ++l) {
    const T xl = shfl(l < 32 ? x0 : x1, l & 31);
    if (lane > l && lane < kb) x0 = sub(x0, mul(L[l * kb + lane], xl));
    if (lane + 32 > l && lane + 32 < kb) x1 = sub(x1, mul(L[l * kb + lane + 32], xl));
  }
  T *out = rhs ? X + (std::size_t)(ci - nright) * ldx : col;
  if (lane < kb) out[k + lane] = x0;
  if (lane + 32 < kb) out[k + lane + 32] = x1;
}

__global__ void iota_kernel(int n, int *p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = i;
}

// X(i, c) = B(perm[i], c)
template <typename T>
__global__ void gather_rows_kernel(int n, int nrhs, const int *__restrict__ perm,
                                   const T *__restrict__ B, int ldb, T *__restrict__ X, int ldx) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n) return;
  const int src = perm[row];
  for (int c = blockIdx.y; c < nrhs; c += gridDim.y)
    X[(std::size_t)c * ldx + row] = B[(std::size_t)c * ldb + src];
}

// The same solve for a full block (kb = 32 VPL): the steps run in runs of 32
// whose pivot rows sit in one register of every lane (x[vo]), so the lane
// selection and most bound checks are static; each row still takes the
// updates in the same order, so the results are those of the general kernel.
template <typename T, bool LOWER, int VPL>
__global__ void __launch_bounds__(256)
    trsm_diag_full_kernel(int nrhs, const T *__restrict__ LU, int lda, int k, T *__restrict__ X, int ldx) {
  constexpr int kb = 32 * VPL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *D = reinterpret_cast<T *>(smem_raw);
  T *rdiag = D + kb * kb;
  load_diag_block(D, LU, lda, k, kb);
  __syncthreads();
  if (!LOWER && threadIdx.x < kb) {
    const T d = D[threadIdx.x * kb + threadIdx.x];
    rdiag[threadIdx.x] = divide(elem<T>::one(), d);
  }
  __syncthreads();
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * warps + (threadIdx.x >> 5);
  if (c >= nrhs) return;
  T *col = X + (std::size_t)c * ldx + k;
  T x[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) x[v] = col[lane + 32 * v];
  if (LOWER) {
#pragma unroll
    for (int vo = 0; vo < VPL; ++vo) {
#pragma unroll 4
      for (int ll = 0; ll < 32; ++ll) {
        const int l = 32 * vo + ll;
        const T xl = shfl(x[vo], ll);
        if (lane > ll) x[vo] = sub(x[vo], mul(D[l * kb + lane + 32 * vo], xl));
#pragma unroll
        for (int v = vo + 1; v < VPL; ++v) x[v] = sub(x[v], mul(D[l * kb + lane + 32 * v], xl));
      }
    }
  } else {
#pragma unroll
    for (int vo = VPL - 1; vo >= 0; --vo) {
#pragma unroll 4
      for (int ll = 31; ll >= 0; --ll) {
        const int l = 32 * vo + ll;
        const T xl = mul(shfl(x[vo], ll), rdiag[l]);
        if (lane == ll) x[vo] = xl;
        if (lane < ll) x[vo] = sub(x[vo], mul(D[l * kb + lane + 32 * vo], xl));
#pragma unroll
        for (int v = 0; v < vo; ++v) x[v] = sub(x[v], mul(D[l * kb + lane + 32 * v], xl));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < VPL; ++v) col[lane + 32 * v] = x[v];
}

// Diagonal-block triangular solve on rows [k, k+kb) of X (kb <= 32 VPL), one
// warp per RHS column, lane l keeping rows l, l + 32, ... LOWER: unit lower
// (forward); else non-unit upper (backward), whose diagonal reciprocals are
// formed once per block, off the dependent chain.
template <typename T, bool LOWER, int VPL>
__global__ void __launch_bounds__(256)
    trsm_diag_kernel(int nrhs, const T *__restrict__ LU, int lda, int k, int kb, T *__restrict__ X,
                     int ldx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *D = reinterpret_cast<T *>(smem_raw);
  T *rdiag = D + kb * kb;
  load_diag_block(D, LU, lda, k, kb);
  __syncthreads();
  if (!LOWER && threadIdx.x < kb) {
    const T d = D[threadIdx.x * kb + threadIdx.x];
    rdiag[threadIdx.x] = divide(elem<T>::one(), d);
  }
  __syncthreads();
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * warps + (threadIdx.x >> 5);
  if (c >= nrhs) return;
  T *col = X + (std::size_t)c * ldx + k;
  T x[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) x[v] = lane + 32 * v < kb ? col[lane + 32 * v] : elem<T>::zero();
  if (LOWER) {
    for (int l = 0; l < kb; ++l) {
      T src = x[0];
#pragma unroll
      for (int v = 1; v < VPL; ++v)
        if ((l >> 5) == v) src = x[v];
      const T xl = shfl(src, l & 31);
#pragma unroll
      for (int v = 0; v < VPL; ++v)
        if (lane + 32 * v > l && lane + 32 * v < kb) x[v] = sub(x[v], mul(D[l * kb + lane + 32 * v], xl));
    }
  } else {
    for (int l = kb - 1; l >= 0; --l) {
      T src = x[0];
#pragma unroll
      for (int v = 1; v < VPL; ++v)
        if ((l >> 5) == v) src = x[v];
      const T xl = mul(shfl(src, l & 31), rdiag[l]);
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        if (lane + 32 * v == l) x[v] = xl;
        if (lane + 32 * v < l) x[v] = sub(x[v], mul(D[l * kb + lane + 32 * v], xl));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < VPL; ++v)
    if (lane + 32 * v < kb) col[lane + 32 * v] = x[v];
}

// Configurations of the one-row-per-thread panel: KB columns (a row's elements
// in registers, the multipliers' KB columns in shared memory), at most MAXT
// threads per CTA. Float and double and complex64 rows take 64 registers;
// complex128 panels of up to 2048 rows run 32 columns (128 registers, 256
// threads): 57 us against two times 27 us with 16 columns at 1024 rows, and half
// as many swap and update launches between panels.
template <typename T> struct RowsPanel;
template <> struct RowsPanel<float> { static constexpr int KB = 64, MAXT = 512, KBs = 64, MAXTs = 512; };
template <> struct RowsPanel<double> { static constexpr int KB = 32, MAXT = 512, KBs = 32, MAXTs = 512; };
template <> struct RowsPanel<float2> { static constexpr int KB = 32, MAXT = 512, KBs = 32, MAXTs = 512; };
template <> struct RowsPanel<double2> { static constexpr int KB = 16, MAXT = 512, KBs = 32, MAXTs = 256; };
constexpr int kRowsMax = kPanelMaxCluster * 512;  // tallest panel of that kernel
template <typename T> constexpr int short_rows() { return kPanelMaxCluster * RowsPanel<T>::MAXTs; }

// Panel width for an n x n factorisation: that of the one-row-per-thread
// panel; beyond its tallest panel, the widest whose full-height panel fits in
// kMaxCluster CTAs' shared memory (lu_panel_kernel).
template <typename T>
int choose_kb(int n) {
  if (n <= short_rows<T>()) return RowsPanel<T>::KBs;
  int kb = RowsPanel<T>::KB;
  while (kb > 1 && n > kRowsMax && (std::size_t)n * kb * sizeof(T) > kPanelSmemBudget * kMaxCluster) kb /= 2;
  return kb;
}

inline cudaLaunchAttribute cluster_attr(int ncta) {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeClusterDimension;
  a.val.clusterDim.x = ncta;
  a.val.clusterDim.y = 1;
  a.val.clusterDim.z = 1;
  return a;
}

// One row per thread: one CTA up to MAXT rows (512; 256 for complex128 factorisations
// of n <= 2048), where the exchange between CTAs costs more than the warps that share
// an SM (a float64 column of 512 rows: 1.09 us in one CTA, 1.22 to 1.28 in 2 to 8);
// above, always eight CTAs, since fewer rows per SM shorten the update (float64,
// 2048 rows: 1.54 us a column on four CTAs, 1.37 on eight).
template <typename T, int KB, int MAXT>
cudaError_t launch_rows_panel(cudaStream_t s, int n, T *A, int lda, int k, int kb, const LuScratch &sc,
                              const RowMap &map, int *info, const PanelWait &wait) {
  const int h = n - k;
  const int ncta = h <= MAXT ? 1 : kPanelMaxCluster;
  int nt = ((h + ncta - 1) / ncta + 31) / 32 * 32;
  if (nt < 64) nt = 64;  // the threads that list the rows moved down: kb <= 64
  auto kern = lu_panel_rows_kernel<T, KB, MAXT>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)panel_rows_smem<T, KB>(MAXT));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncta, 1, 1);
  cfg.blockDim = dim3(nt, 1, 1);
  cfg.dynamicSmemBytes = panel_rows_smem<T, KB>(nt);
  cfg.stream = s;
  cudaLaunchAttribute attr[1] = {cluster_attr(ncta)};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, kern, n, A, lda, k, kb, sc.ipiv, sc.perm, map.pos, map.src, map.count, info, wait);
}

template <typename T>
cudaError_t launch_panel(cudaStream_t s, int n, T *A, int lda, int k, int kb, const LuScratch &sc,
                         const RowMap &map, int *info, const PanelWait &wait) {
  const int h = n - k;
  using C = RowsPanel<T>;
  if (n <= short_rows<T>()) return launch_rows_panel<T, C::KBs, C::MAXTs>(s, n, A, lda, k, kb, sc, map, info, wait);
  if (h <= kRowsMax) return launch_rows_panel<T, C::KB, C::MAXT>(s, n, A, lda, k, kb, sc, map, info, wait);
  // enough CTAs for the panel to fit, and for every row to get >= 2 lanes of
  // the fused pass when the cluster allows it (<= 256 rows per CTA)
  int ncta = (int)(((std::size_t)h * kb * sizeof(T) + kPanelSmemBudget - 1) / kPanelSmemBudget);
  const int by_rows = (h + 255) / 256;
  if (ncta < by_rows) ncta = by_rows;
  if (ncta < 1) ncta = 1;
  if (ncta > kMaxCluster) ncta = kMaxCluster;
  if (ncta > h) ncta = h;
  const int rpc = (h + ncta - 1) / ncta;
  const PanelSmem o = panel_smem<T>(rpc, kb);
  auto kern = lu_panel_kernel<T>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)o.total);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncta, 1, 1);
  // threads: enough lanes for every row x column phase, in whole warps
  int ncph = 1;
  while (ncph * 2 <= 32 && ncph * 2 * rpc <= kPanelThreads) ncph *= 2;
  int nt = ((rpc * ncph + 31) / 32) * 32;
  if (nt > kPanelThreads) nt = kPanelThreads;
  if (nt < 64) nt = 64;
  cfg.blockDim = dim3(nt, 1, 1);
  cfg.dynamicSmemBytes = o.total;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, kern, n, A, lda, k, kb, rpc, sc.ipiv, sc.perm, map.pos, map.src, map.count,
                            info);
}

}  // namespace

std::size_t lu_scratch_bytes(int n) {
  Layout L(nullptr);
  L.take<int>(n < 1 ? 1 : n);  // ipiv
  L.take<int>(n < 1 ? 1 : n);  // perm
  for (int i = 0; i < 2; ++i) {  // the row maps
    L.take<int>(2 * kMaxKb);
    L.take<int>(2 * kMaxKb);
    L.take<int>(1);
  }
  return L.used;
}

// Look-ahead resources of the calling host thread on the current device: a
// high-priority auxiliary stream on which the next panel is factored while the
// caller's stream runs the wide trailing update, and the two events that order
// them.
struct LookAhead {
  int device = -1;
  cudaStream_t aux = nullptr;
  cudaEvent_t ready = nullptr, done = nullptr;
};
thread_local LookAhead tl_lookahead;
thread_local bool tl_no_lookahead = false;

cudaError_t lookahead(LookAhead *&out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  LookAhead &la = tl_lookahead;
  if (la.device != dev) {
    if (la.aux) {  // a different device than last time: release the old set
      cudaStreamDestroy(la.aux);
      cudaEventDestroy(la.ready);
      cudaEventDestroy(la.done);
      la = LookAhead{};
    }
    int lo = 0, hi = 0;
    if ((e = cudaDeviceGetStreamPriorityRange(&lo, &hi)) != cudaSuccess) return e;
    if ((e = cudaStreamCreateWithPriority(&la.aux, cudaStreamNonBlocking, hi)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&la.ready, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&la.done, cudaEventDisableTiming)) != cudaSuccess) return e;
    la.device = dev;
  }
  out = &la;
  return cudaSuccess;
}

// Blocked right-looking factorisation with a one-panel look-ahead. The panel
// is a latency chain on at most eight SMs, so what it waits for comes first:
// after panel k, the swaps, U12 and the update of the next panel's columns
// alone; then panel k+1 runs on the auxiliary stream while the caller's stream
// does the same for the other columns. With a right-hand side (B != null) its
// forward substitution is part of that: B's columns take the swaps, the solve
// with L11 and the update like the matrix's own, in the time that the caller's
// stream would wait for the panels, and X receives L^-1 P B; B is overwritten.
// The columns left of a panel take its swaps (keep_l) only where L is used
// again. Forward substitution after the factorisation, against this: complex128
// 1024 expm 4986 -> 4638 us, float64 1501 5555 -> 5035, float32 4096 15478 ->
// 12918 (with the split inside its updates), complex64 777 3123 -> 2591.
template <typename T>
static cudaError_t factor(cudaStream_t s, int n, T *A, int lda, const LuScratch &sc, int *info_dev, bool keep_l,
                          int nrhs, T *B, int ldb, T *X, int ldx, const PanelWait &wait = {}) {
  cudaError_t e = cudaMemsetAsync(info_dev, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  iota_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, sc.perm);
  if ((e = launched()) != cudaSuccess) return e;
  const int kbn = choose_kb<T>(n);
  auto swap_kern = lu_swap_trsm_kernel<T>;
  const std::size_t swap_smem = sizeof(T) * (std::size_t)kbn * kbn;
  if ((e = cudaFuncSetAttribute(swap_kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)swap_smem)) !=
      cudaSuccess)
    return e;
  // only matrices of more than one panel use the look-ahead stream, and not
  // while a NoLookAheadScope is open on this thread (then every panel runs on s)
  const bool ahead = n > kbn && !tl_no_lookahead;
  LookAhead *la = nullptr;
  if (ahead && (e = lookahead(la)) != cudaSuccess) return e;
  if ((e = launch_panel<T>(s, n, A, lda, 0, kbn < n ? kbn : n, sc, sc.map[0], info_dev, wait)) != cudaSuccess) return e;
  for (int k = 0, step = 0; k < n; k += kbn, ++step) {
    const int kb = (k + kbn < n) ? kbn : n - k;
    const RowMap &map = sc.map[step & 1];
    if (ahead && k > 0 && (e = cudaStreamWaitEvent(s, la->done, 0)) != cudaSuccess) return e;  // panel k
    // swaps and solve of nright columns from c0 on, of the right-hand side, and swaps of nleft columns
    auto swaps = [&](int c0, int nright, int rhs, int nleft) -> cudaError_t {
      const int cols = nright + rhs + nleft;
      if (cols == 0) return cudaSuccess;
      const int warps = 8;
      swap_kern<<<(cols + warps - 1) / warps, warps * 32, sizeof(T) * (std::size_t)kb * kb, s>>>(
          A, lda, k, kb, c0, nright, nleft, B, ldb, X, ldx, rhs, map.pos, map.src, map.count);
      return launched();
    };
    const int rest = n - (k + kb);
    const int kb2 = rest < kbn ? rest : kbn;  // the next panel's width
    const T *L21 = A + (std::size_t)k * lda + (k + kb);
    auto update = [&](const T *U, int ldu, T *C, int ldc, int cols) -> cudaError_t {
      if (rest == 0 || cols == 0) return cudaSuccess;
      return gemm_nn<T>(s, rest, cols, kb, -1.0, L21, lda, U, ldu, 1.0, C, ldc);
    };
    if (rest > 0) {  // the next panel's columns first
      T *next = A + (std::size_t)(k + kb) * lda + k;
      if ((e = swaps(k + kb, kb2, 0, 0)) != cudaSuccess) return e;
      if ((e = update(next, lda, next + kb, lda, kb2)) != cudaSuccess) return e;
      if (ahead) {
        if ((e = cudaEventRecord(la->ready, s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(la->aux, la->ready, 0)) != cudaSuccess) return e;
        if ((e = launch_panel<T>(la->aux, n, A, lda, k + kb, kb2, sc, sc.map[(step + 1) & 1], info_dev, wait)) !=
            cudaSuccess)
          return e;
        if ((e = cudaEventRecord(la->done, la->aux)) != cudaSuccess) return e;
      } else if ((e = launch_panel<T>(s, n, A, lda, k + kb, kb2, sc, sc.map[(step + 1) & 1], info_dev, wait)) !=
                 cudaSuccess) {  // disjoint from the other columns
        return e;
      }
    }
    // the other columns, concurrent with that panel
    const int c1 = k + kb + kb2;
    if ((e = swaps(c1, n - c1, nrhs, keep_l ? k : 0)) != cudaSuccess) return e;
    T *U = A + (std::size_t)c1 * lda + k;
    if ((e = update(U, lda, U + kb, lda, n - c1)) != cudaSuccess) return e;
    if (nrhs > 0 && (e = update(X + k, ldx, B + k + kb, ldb, nrhs)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t getrf(cudaStream_t s, int n, T *A, int lda, void *scratch, int *info_dev, PanelWait wait) {
  if (n < 1) return cudaSuccess;
  return factor<T>(s, n, A, lda, carve_lu(scratch, n), info_dev, true, 0, nullptr, 0, nullptr, 0, wait);
}

// X <- L^-1 X (lower) and X <- U^-1 X (upper) by diagonal blocks.
template <typename T>
static cudaError_t triangular_solves(cudaStream_t s, int n, int nrhs, const T *LU, int lda, T *X, int ldx, bool lower,
                                     bool upper) {
  cudaError_t e;
  // Diagonal blocks of 64 rows; float32 systems above 1024 take 128 (half as
  // many passes of the off-diagonal updates over the right-hand side: float32
  // 4096 expm +3 %; float64 2048 measured 8 % slower with 128)
  const bool wide = std::is_same<T, float>::value && n > 1024;
  const int NB = wide ? 128 : 64;
  const int warps = 8;
  const std::size_t smem = sizeof(T) * (NB * NB + NB);
  auto kl = wide ? trsm_diag_kernel<T, true, 4> : trsm_diag_kernel<T, true, 2>;
  auto ku = wide ? trsm_diag_kernel<T, false, 4> : trsm_diag_kernel<T, false, 2>;
  // full blocks (every one but a ragged last) take the static-lane kernel
  auto fl = wide ? trsm_diag_full_kernel<T, true, 4> : trsm_diag_full_kernel<T, true, 2>;
  auto fu = wide ? trsm_diag_full_kernel<T, false, 4> : trsm_diag_full_kernel<T, false, 2>;
  for (auto kern : {kl, ku})
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
      return e;
  for (auto kern : {fl, fu})
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
      return e;
  const int blocks = (nrhs + warps - 1) / warps;
  for (int k = 0; lower && k < n; k += NB) {
    const int kb = (k + NB < n) ? NB : n - k;
    if (kb == NB) fl<<<blocks, warps * 32, sizeof(T) * (kb * kb + kb), s>>>(nrhs, LU, lda, k, X, ldx);
    else kl<<<blocks, warps * 32, sizeof(T) * (kb * kb + kb), s>>>(nrhs, LU, lda, k, kb, X, ldx);
    if ((e = launched()) != cudaSuccess) return e;
    if (k + kb < n) {
      e = gemm_nn<T>(s, n - (k + kb), nrhs, kb, -1.0, LU + (std::size_t)k * lda + (k + kb), lda,
                     X + k, ldx, 1.0, X + (k + kb), ldx);
      if (e != cudaSuccess) return e;
    }
  }
  const int last = ((n - 1) / NB) * NB;
  for (int k = last; upper && k >= 0; k -= NB) {
    const int kb = (k + NB < n) ? NB : n - k;
    if (kb == NB) fu<<<blocks, warps * 32, sizeof(T) * (kb * kb + kb), s>>>(nrhs, LU, lda, k, X, ldx);
    else ku<<<blocks, warps * 32, sizeof(T) * (kb * kb + kb), s>>>(nrhs, LU, lda, k, kb, X, ldx);
    if ((e = launched()) != cudaSuccess) return e;
    if (k > 0) {
      e = gemm_nn<T>(s, k, nrhs, kb, -1.0, LU + (std::size_t)k * lda, lda, X + k, ldx, 1.0, X, ldx);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t getrf_solve(cudaStream_t s, int n, T *A, int lda, void *scratch, int nrhs, T *B, int ldb, T *X, int ldx,
                        bool keep_l, int *info_dev) {
  if (n < 1) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(info_dev + 1, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  if ((e = factor<T>(s, n, A, lda, carve_lu(scratch, n), info_dev, keep_l, nrhs, B, ldb, X, ldx)) != cudaSuccess)
    return e;
  return triangular_solves<T>(s, n, nrhs, A, lda, X, ldx, false, true);
}

template <typename T>
cudaError_t getrs(cudaStream_t s, int n, int nrhs, const T *LU, int lda, const void *scratch,
                  const T *B, int ldb, T *X, int ldx, int *info_dev) {
  if (n < 1 || nrhs < 1) return cudaSuccess;
  const LuScratch sc = carve_lu(const_cast<void *>(scratch), n);
  cudaError_t e = cudaMemsetAsync(info_dev, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  {
    const int gy = nrhs < 65535 ? nrhs : 65535;
    gather_rows_kernel<T><<<dim3((n + 255) / 256, gy), 256, 0, s>>>(n, nrhs, sc.perm, B, ldb, X, ldx);
    if ((e = launched()) != cudaSuccess) return e;
  }
  return triangular_solves<T>(s, n, nrhs, LU, lda, X, ldx, true, true);
}

#define CLM_INST_LU(T)                                                                            \
  template cudaError_t getrf<T>(cudaStream_t, int, T *, int, void *, int *, PanelWait);          \
  template cudaError_t getrs<T>(cudaStream_t, int, int, const T *, int, const void *, const T *, \
                                int, T *, int, int *);                                           \
  template cudaError_t getrf_solve<T>(cudaStream_t, int, T *, int, void *, int, T *, int, T *, int, bool, int *);
CLM_INST_LU(float)
CLM_INST_LU(double)
CLM_INST_LU(float2)
CLM_INST_LU(double2)
#undef CLM_INST_LU

}  // namespace clm
