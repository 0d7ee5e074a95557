// batched.cu -- expm of many small matrices (n <= 256) in one call.
//
// New entry point (calaman_G evaluates one matrix per call): every matrix of
// the batch gets its own (m, s) from its own 1-norm, exactly as expm would
// pick, and the whole batch advances phase by phase -- one kernel launch per
// phase covers every matrix, whatever its size and degree:
//
//   norm -> (one readback, plans on the host) -> scale -> A2 -> A4 -> A6 -> A8
//   -> even/odd combinations -> [m = 13: W += A6 T, V += A6 Z] -> U = X W
//   -> p = V + U, q = V - U -> LU(q) + solve (fused, one CTA per matrix)
//   -> s squarings (FP64 for the single tier) -> write-back
//
// Each kernel reads a per-matrix descriptor table (pointers, n, ld, plan) and
// derives its own operands, so a phase in which a matrix takes no part costs
// that matrix nothing but an early exit. The dense products run on a grouped
// GEMM: one CTA per 64 x 64 output tile, tiles of all matrices numbered
// consecutively, each CTA finding its matrix by binary search on the tile
// prefix sums. The LU and the n-right-hand-side solve of a matrix run in one
// CTA of 256 threads in which thread i owns row i (pivot search, swaps,
// rank-updates) or column i (swap gathers, triangular solves of the diagonal
// blocks), with panels of 32 columns.
#include <algorithm>
#include <cfloat>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>

#include "dmma.cuh"
#include "expm_common.cuh"
#include "tcgen05.cuh"

namespace clm {
namespace {

constexpr int kBatchedMaxN = 256;
constexpr int kBThreads = 256;  // = kBatchedMaxN: one thread per row / column
constexpr int kBPanel = 32;
constexpr int kGTile = 64;      // grouped GEMM output tile
constexpr int kGK = 16;         // grouped GEMM k-chunk
constexpr int kEwChunk = 16384; // elements per elementwise CTA

// Per-matrix buffers (ld = n): X (scaled input, later the Pade quotient),
// P0..P3 (even powers; P0 is also U and p), T (m = 13 odd temp), V, W, and
// for the squarings two buffers of the wide type.
template <typename T, typename Wd>
struct BItem {
  const T *A;
  T *E;
  T *X, *P0, *P1, *P2, *P3, *Tt, *V, *W;
  Wd *wa, *wb;
  int n, lda, lde, id;  // id: the matrix's index in the caller's batch (d_info)
};

struct BPlan {
  int m, s, np, pad;
};

enum BPhase { kPhA2 = 0, kPhA4, kPhA6, kPhA8, kPhM13, kPhU, kPhSq };

// Pade coefficients b_0..b_13 of each degree, indexed by (m - 3) / 2 for
// m < 13 and 4 for m = 13.
__constant__ double c_pade[5][14];

template <typename To> __device__ __forceinline__ To convert_elem(float x);
template <> __device__ __forceinline__ float convert_elem<float>(float x) { return x; }
template <> __device__ __forceinline__ double convert_elem<double>(float x) { return (double)x; }
template <typename To> __device__ __forceinline__ To convert_elem(double x);
template <> __device__ __forceinline__ double convert_elem<double>(double x) { return x; }
template <> __device__ __forceinline__ float convert_elem<float>(double x) { return (float)x; }

__device__ __forceinline__ float conj_elem(float x) { return x; }
__device__ __forceinline__ double conj_elem(double x) { return x; }

__device__ __forceinline__ int degree_slot(int m) { return m == 13 ? 4 : (m - 3) / 2; }

// ---- 1-norm of every matrix: one CTA per matrix --------------------------
template <typename Item>
__global__ void __launch_bounds__(256) b_norm_kernel(const Item *__restrict__ items,
                                                     double *__restrict__ norms) {
  const Item it = items[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double best = 0.0;
  bool nan = false;
  for (int c = warp; c < it.n; c += 8) {
    double sum = 0.0;
    for (int r = lane; r < it.n; r += 32) sum += modulus(it.A[(std::size_t)c * it.lda + r]);
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    nan |= sum != sum;
    best = fmax(best, sum);
  }
  __shared__ double red[8];
  __shared__ int red_nan[8];
  if (lane == 0) {
    red[warp] = best;
    red_nan[warp] = nan;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    int anynan = 0;
    for (int w = 0; w < 8; ++w) {
      b = fmax(b, red[w]);
      anynan |= red_nan[w];
    }
    norms[blockIdx.x] = anynan ? (double)NAN : b;
  }
}

// ---- elementwise phases: CTA (chunk, matrix) ------------------------------
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) b_scale_kernel(const BItem<T, Wd> *__restrict__ items,
                                                      const BPlan *__restrict__ plans) {
  using R = typename elem<T>::real;
  const BPlan pl = plans[blockIdx.x];
  if (pl.s == 0) return;
  const BItem<T, Wd> it = items[blockIdx.x];
  const int nn = it.n * it.n;
  const R f = (R)ldexp(1.0, -pl.s);
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    const int c = e / it.n, r = e - c * it.n;
    it.X[e] = scale(it.A[(std::size_t)c * it.lda + r], f);
  }
}

// W consecutive elements, moved as one 16-byte piece where W fills it. The
// elementwise phases below are bound by memory and by the loads in flight: where
// a matrix's n^2 is a multiple of the piece (ld = n) and its buffers are aligned,
// a thread takes a piece per step, else one element.
template <typename T> constexpr int ew_piece() { return 16 / (int)sizeof(T); }
template <int W, typename T>
struct Pack {
  T e[W];
};
template <int W, typename T>
__device__ __forceinline__ Pack<W, T> ew_load(const T *p) {
  Pack<W, T> v;
  if constexpr (W > 1) {
    union {
      uint4 u;
      T e[W];
    } w;
    w.u = *reinterpret_cast<const uint4 *>(p);
#pragma unroll
    for (int i = 0; i < W; ++i) v.e[i] = w.e[i];
  } else {
    v.e[0] = *p;
  }
  return v;
}
template <int W, typename T>
__device__ __forceinline__ void ew_store(T *p, const Pack<W, T> &v) {
  if constexpr (W > 1) {
    union {
      uint4 u;
      T e[W];
    } w;
#pragma unroll
    for (int i = 0; i < W; ++i) w.e[i] = v.e[i];
    *reinterpret_cast<uint4 *>(p) = w.u;
  } else {
    *p = v.e[0];
  }
}
// body(std::integral_constant<int, W>, e) for every piece of this CTA's chunk of
// nn elements; buf: one of the matrix's buffers, which all lie 256 bytes apart
template <typename T, typename F>
__device__ __forceinline__ void ew_for(const T *buf, int nn, F &&body) {
  constexpr int V = ew_piece<T>();
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  if (nn % V == 0 && (reinterpret_cast<std::uintptr_t>(buf) & 15) == 0) {
    for (int e = blockIdx.y * kEwChunk + threadIdx.x * V; e < end; e += blockDim.x * V)
      body(std::integral_constant<int, V>{}, e);
  } else {
    for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x)
      body(std::integral_constant<int, 1>{}, e);
  }
}
// body(i, diagonal) for the elements e .. e + W - 1 of an n x n matrix
template <int W, typename F>
__device__ __forceinline__ void ew_diag(int e, int n, F &&body) {
  int c = e / n, r = e - c * n;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    body(i, r == c);
    if (++r == n) r = 0, ++c;
  }
}

// V, W from the even powers (m < 13); for m = 13 also the odd temp T and the
// even temp (into P3, unused at m = 13):
//   T = b9 A2 + b11 A4 + b13 A6,  W = b1 I + b3 A2 + b5 A4 + b7 A6,
//   Z = b8 A2 + b10 A4 + b12 A6,  V = b0 I + b2 A2 + b4 A4 + b6 A6.
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) b_even_odd_kernel(const BItem<T, Wd> *__restrict__ items,
                                                         const BPlan *__restrict__ plans) {
  using R = typename elem<T>::real;
  const BItem<T, Wd> it = items[blockIdx.x];
  const BPlan pl = plans[blockIdx.x];
  const double *b = c_pade[degree_slot(pl.m)];
  const int n = it.n;
  const T *P[4] = {it.P0, it.P1, it.P2, it.P3};
  ew_for<T>(it.V, n * n, [&](auto piece, int e) {
    constexpr int W = decltype(piece)::value;
    if (pl.m != 13) {
      Pack<W, T> v, w;
#pragma unroll
      for (int i = 0; i < W; ++i) v.e[i] = w.e[i] = elem<T>::zero();
      for (int k = 0; k < pl.np; ++k) {
        const Pack<W, T> x = ew_load<W>(P[k] + e);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          v.e[i] = rfma((R)b[2 * k + 2], x.e[i], v.e[i]);
          w.e[i] = rfma((R)b[2 * k + 3], x.e[i], w.e[i]);
        }
      }
      ew_diag<W>(e, n, [&](int i, bool diag) {
        if (diag) {
          v.e[i] = add_real(v.e[i], (R)b[0]);
          w.e[i] = add_real(w.e[i], (R)b[1]);
        }
      });
      ew_store<W>(it.V + e, v);
      ew_store<W>(it.W + e, w);
    } else {
      const Pack<W, T> x1 = ew_load<W>(it.P0 + e), x2 = ew_load<W>(it.P1 + e), x3 = ew_load<W>(it.P2 + e);
      Pack<W, T> t, w, z, v;
#pragma unroll
      for (int i = 0; i < W; ++i) {
        t.e[i] = rfma((R)b[13], x3.e[i], rfma((R)b[11], x2.e[i], scale(x1.e[i], (R)b[9])));
        w.e[i] = rfma((R)b[7], x3.e[i], rfma((R)b[5], x2.e[i], scale(x1.e[i], (R)b[3])));
        z.e[i] = rfma((R)b[12], x3.e[i], rfma((R)b[10], x2.e[i], scale(x1.e[i], (R)b[8])));
        v.e[i] = rfma((R)b[6], x3.e[i], rfma((R)b[4], x2.e[i], scale(x1.e[i], (R)b[2])));
      }
      ew_diag<W>(e, n, [&](int i, bool diag) {
        if (diag) {
          w.e[i] = add_real(w.e[i], (R)b[1]);
          v.e[i] = add_real(v.e[i], (R)b[0]);
        }
      });
      ew_store<W>(it.Tt + e, t);
      ew_store<W>(it.W + e, w);
      ew_store<W>(it.P3 + e, z);
      ew_store<W>(it.V + e, v);
    }
  });
}

// p = V + U over P0 (which holds U), q = V - U over V
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) b_split_kernel(const BItem<T, Wd> *__restrict__ items) {
  const BItem<T, Wd> it = items[blockIdx.x];
  ew_for<T>(it.V, it.n * it.n, [&](auto piece, int e) {
    constexpr int W = decltype(piece)::value;
    const Pack<W, T> u = ew_load<W>(it.P0 + e), v = ew_load<W>(it.V + e);
    Pack<W, T> p, q;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      p.e[i] = add(v.e[i], u.e[i]);
      q.e[i] = sub(v.e[i], u.e[i]);
    }
    ew_store<W>(it.P0 + e, p);
    ew_store<W>(it.V + e, q);
  });
}

// s > 0: wa = (Wd) X, the Pade quotient
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) b_widen_kernel(const BItem<T, Wd> *__restrict__ items,
                                                      const BPlan *__restrict__ plans) {
  if (plans[blockIdx.x].s == 0) return;
  const BItem<T, Wd> it = items[blockIdx.x];
  const int nn = it.n * it.n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x)
    it.wa[e] = convert_elem<Wd>(it.X[e]);
}

// s > 0: E = (T) the last square (wa for even s, wb for odd s)
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) b_narrow_kernel(const BItem<T, Wd> *__restrict__ items,
                                                       const BPlan *__restrict__ plans) {
  const int s = plans[blockIdx.x].s;
  if (s == 0) return;
  const BItem<T, Wd> it = items[blockIdx.x];
  const Wd *src = (s & 1) ? it.wb : it.wa;
  const int n = it.n, nn = n * n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    const int c = e / n, r = e - c * n;
    it.E[(std::size_t)c * it.lde + r] = convert_elem<T>(src[e]);
  }
}

// ---- grouped GEMM: C (+)= +-(A B [+ A2 B2]), n x n x n per matrix, one 64 x 64
// output tile per CTA. What a phase multiplies is decided per matrix by an
// operand policy (Ops::pade for the evaluation phases, Ops::square for the
// squarings); blockIdx.y selects a sub-problem of the phase.
// four consecutive shared-memory elements (src 16-byte aligned)
template <typename T>
__device__ __forceinline__ void lds4(const T *src, T (&dst)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4 *>(src);
    dst[0] = v.x, dst[1] = v.y, dst[2] = v.z, dst[3] = v.w;
  } else if constexpr (sizeof(T) == 8) {
    const double2 *s2 = reinterpret_cast<const double2 *>(src);
    union { double2 v[2]; T e[4]; } u;
    u.v[0] = s2[0];
    u.v[1] = s2[1];
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = u.e[i];
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = src[i];
  }
}

template <typename U>
struct GOps {
  const U *A = nullptr, *B = nullptr, *A2 = nullptr, *B2 = nullptr;
  U *C = nullptr;
  int lda = 0, ldb = 0, lda2 = 0, ldb2 = 0, ldc = 0;
  bool acc = false, neg = false;
};

// expm: the evaluation phases and the squarings of BItem matrices
struct ExpmOps {
  template <typename T, typename Wd>
  static __device__ __forceinline__ bool pade(const BItem<T, Wd> &it, const BPlan &pl, int phase, int sub,
                                              GOps<T> &o) {
    const T *X = pl.s > 0 ? it.X : it.A;
    const int ldx = pl.s > 0 ? it.n : it.lda;
    o.lda = o.ldb = o.ldc = it.n;
    switch (phase) {
    case kPhA2:
      o.A = X; o.lda = ldx; o.B = X; o.ldb = ldx; o.C = it.P0;
      return true;
    case kPhA4:
      o.A = it.P0; o.B = it.P0; o.C = it.P1;
      return pl.np >= 2;
    case kPhA6:
      o.A = it.P1; o.B = it.P0; o.C = it.P2;
      return pl.np >= 3;
    case kPhA8:
      o.A = it.P1; o.B = it.P1; o.C = it.P3;
      return pl.np >= 4;
    case kPhM13:
      o.A = it.P2; o.B = sub ? it.P3 : it.Tt; o.C = sub ? it.V : it.W; o.acc = true;
      return pl.m == 13;
    case kPhU:
      o.A = X; o.lda = ldx; o.B = it.W; o.C = it.P0;
      return true;
    default:
      return false;
    }
  }
  // square k reads wa for odd k, wb for even k
  template <typename T, typename Wd>
  static __device__ __forceinline__ bool square(const BItem<T, Wd> &it, const BPlan &pl, int sub, int k,
                                                GOps<Wd> &o) {
    o.A = o.B = (k & 1) ? it.wa : it.wb;
    o.C = (k & 1) ? it.wb : it.wa;
    o.lda = o.ldb = o.ldc = it.n;
    return pl.s >= k && sub == 0;
  }
};

template <typename Item, typename U, typename Ops, bool kSquare>
__global__ void __launch_bounds__(256)
    g_gemm_kernel(const Item *__restrict__ items, const BPlan *__restrict__ plans,
                  const int *__restrict__ tile_prefix, int batch, int phase, int ksq) {
  // the matrix of this tile: last i with tile_prefix[i] <= blockIdx.x
  const int tile = blockIdx.x;
  int lo = 0, hi = batch - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_prefix[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  const Item it = items[lo];
  const BPlan pl = plans[lo];
  GOps<U> o;
  if constexpr (kSquare) {
    if (!Ops::square(it, pl, blockIdx.y, ksq, o)) return;
  } else {
    if (!Ops::pade(it, pl, phase, blockIdx.y, o)) return;
  }
  const int n = it.n;
  const int tn = (n + kGTile - 1) / kGTile;
  const int local = tile - tile_prefix[lo];
  const int m0 = (local % tn) * kGTile, n0 = (local / tn) * kGTile;

  __shared__ __align__(16) U As[kGK][kGTile + 4];
  __shared__ __align__(16) U Bs[kGK][kGTile + 4];
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;  // rows 4 tx + i, columns 4 ty + j: one vector load each
  U acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = elem<U>::zero();

  // global -> register staging: A tile (64 rows x 16 k), B tile (16 k x 64 cols)
  const int ar = t & 63, ak = t >> 6;   // A: rows ar, k = ak + 4 q
  const int bk = t & 15, bc = t >> 4;   // B: k = bk, columns bc + 16 q
  const int nprod = o.A2 ? 2 : 1;
  for (int pr = 0; pr < nprod; ++pr) {
    const U *Am = pr ? o.A2 : o.A;
    const U *Bm = pr ? o.B2 : o.B;
    const int lda = pr ? o.lda2 : o.lda, ldb = pr ? o.ldb2 : o.ldb;
    U ra[4], rb[4];
    auto load = [&](int k0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = m0 + ar, k = k0 + ak + 4 * q;
        ra[q] = (r < n && k < n) ? Am[(std::size_t)k * lda + r] : elem<U>::zero();
        const int c = n0 + bc + 16 * q, kb = k0 + bk;
        rb[q] = (c < n && kb < n) ? Bm[(std::size_t)c * ldb + kb] : elem<U>::zero();
      }
    };
    load(0);
    for (int k0 = 0; k0 < n; k0 += kGK) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        As[ak + 4 * q][ar] = ra[q];
        Bs[bk][bc + 16 * q] = rb[q];
      }
      __syncthreads();
      if (k0 + kGK < n) load(k0 + kGK);
#pragma unroll
      for (int kk = 0; kk < kGK; ++kk) {
        U a[4], bv[4];
        lds4(&As[kk][4 * tx], a);
        lds4(&Bs[kk][4 * ty], bv);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmac(a[i], bv[j], acc[i][j]);
      }
    }
  }
  U old[4][4];  // accumulate: every old C value in flight before the first store
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = n0 + 4 * ty + j, r = m0 + 4 * tx + i;
      old[i][j] = (o.acc && c < n && r < n) ? o.C[(std::size_t)c * o.ldc + r] : elem<U>::zero();
    }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = n0 + 4 * ty + j;
    if (c >= n) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = m0 + 4 * tx + i;
      if (r >= n) continue;
      const U v = o.neg ? sub(old[i][j], acc[i][j]) : add(old[i][j], acc[i][j]);
      o.C[(std::size_t)c * o.ldc + r] = v;
    }
  }
}

// ---- grouped FP64 GEMM on the tensor cores (DMMA m16n8k8): the same tile
// numbering, operand policies and epilogue as g_gemm_kernel, with a 64 x 64
// output tile per CTA of four warps (32 x 32 each), k-slices of 16 staged by
// cp.async in a three-stage ring. A second product (A2 B2) continues the same
// k loop into the same accumulators.
constexpr int kDStages = 3;
constexpr int kDSA = kGTile + 4, kDSB = 16 + 4;  // 4 mod 16 doubles: conflict-free fragments
constexpr std::size_t kDSmem = sizeof(double) * kDStages * (16 * kDSA + kGTile * kDSB);

template <typename Item, typename Ops, bool kSquare>
__global__ void __launch_bounds__(128)
    g_dgemm_kernel(const Item *__restrict__ items, const BPlan *__restrict__ plans,
                   const int *__restrict__ tile_prefix, int batch, int phase, int ksq) {
  constexpr int BK = 16, MI = 2, NI = 4;
  const int tile = blockIdx.x;
  int lo = 0, hi = batch - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_prefix[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  const Item it = items[lo];
  const BPlan pl = plans[lo];
  GOps<double> o;
  if constexpr (kSquare) {
    if (!Ops::square(it, pl, blockIdx.y, ksq, o)) return;
  } else {
    if (!Ops::pade(it, pl, phase, blockIdx.y, o)) return;
  }
  const int n = it.n;
  const int tn = (n + kGTile - 1) / kGTile;
  const int local = tile - tile_prefix[lo];
  const int m0 = (local % tn) * kGTile, n0 = (local / tn) * kGTile;

  extern __shared__ __align__(16) double dsm[];
  double *sA = dsm;                                 // [stage][k][m]
  double *sB = dsm + kDStages * BK * kDSA;          // [stage][n][k]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (warp & 1) * 32, wn0 = (warp >> 1) * 32;
  const int KT = (n + BK - 1) / BK;
  const int total = (o.A2 ? 2 : 1) * KT;

  auto load_tile = [&](int stage, int step) {
    const bool second = step >= KT;
    const double *Am = second ? o.A2 : o.A;
    const double *Bm = second ? o.B2 : o.B;
    const int lda = second ? o.lda2 : o.lda, ldb = second ? o.ldb2 : o.ldb;
    const int k0 = (second ? step - KT : step) * BK;
    double *a = sA + stage * BK * kDSA;
    double *b = sB + stage * kGTile * kDSB;
#pragma unroll
    for (int c = tid; c < BK * kGTile; c += 128) {
      const int kk = c / kGTile, mm = c % kGTile;
      const int gm = m0 + mm, gk = k0 + kk;
      const int bytes = (gk < n && gm < n) ? 8 : 0;
      cp_async8(a + kk * kDSA + mm, bytes ? Am + (std::size_t)gk * lda + gm : Am, bytes);
    }
#pragma unroll
    for (int c = tid; c < kGTile * BK; c += 128) {
      const int nn = c / BK, kk = c % BK;
      const int gn = n0 + nn, gk = k0 + kk;
      const int bytes = (gn < n && gk < n) ? 8 : 0;
      cp_async8(b + nn * kDSB + kk, bytes ? Bm + (std::size_t)gn * ldb + gk : Bm, bytes);
    }
  };

  double acc[MI][NI][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;
#pragma unroll
  for (int st = 0; st < kDStages - 1; ++st) {
    if (st < total) load_tile(st, st);
    cp_commit();
  }
  for (int step = 0; step < total; ++step) {
    cp_wait<kDStages - 2>();
    __syncthreads();
    {
      const int nx = step + kDStages - 1;
      if (nx < total) load_tile(nx % kDStages, nx);
      cp_commit();
    }
    const double *a = sA + (step % kDStages) * BK * kDSA;
    const double *b = sB + (step % kDStages) * kGTile * kDSB;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 8) {
      double af[MI][4], bf[NI][2];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int m = wm0 + i * 16 + g;
        af[i][0] = a[(kk + t) * kDSA + m];
        af[i][1] = a[(kk + t) * kDSA + m + 8];
        af[i][2] = a[(kk + t + 4) * kDSA + m];
        af[i][3] = a[(kk + t + 4) * kDSA + m + 8];
      }
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const int nn = wn0 + j * 8 + g;
        bf[j][0] = b[nn * kDSB + kk + t];
        bf[j][1] = b[nn * kDSB + kk + t + 4];
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) dmma16x8x8(acc[i][j], af[i], bf[j]);
    }
  }
  cp_wait<0>();
  // epilogue: all old C values of a row block in flight before any store
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    double old[NI][4];
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = m0 + wm0 + i * 16 + g + ((r & 2) ? 8 : 0);
        const int c = n0 + wn0 + j * 8 + 2 * t + (r & 1);
        old[j][r] = (o.acc && m < n && c < n) ? o.C[(std::size_t)c * o.ldc + m] : 0.0;
      }
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = m0 + wm0 + i * 16 + g + ((r & 2) ? 8 : 0);
        const int c = n0 + wn0 + j * 8 + 2 * t + (r & 1);
        if (m < n && c < n) o.C[(std::size_t)c * o.ldc + m] = o.neg ? old[j][r] - acc[i][j][r]
                                                                    : old[j][r] + acc[i][j][r];
      }
  }
}

// ---- grouped FP32 GEMM on the tcgen05 tensor cores (split-BF16 x6) --------
// One CTA per 128 x 128 output tile of one matrix (tiles of all matrices
// numbered consecutively, as above, with 128-tiles), C (+)= +-(A B [+ A2 B2])
// with the operand policy of the phase. FP32 operands are read straight from
// the matrices (no part buffers): eight producer warps load a 128 x 64 k-block
// of A and of B, split every element into bf16 parts h + m + l and write the
// six part tiles K-major in the 128-byte-swizzled layout tcgen05.mma reads;
// one thread of the ninth warp issues the six part products (l h, h l, m m,
// m h, h m, h h; smallest first) into one FP32 accumulator in TMEM, N = the
// tile's columns rounded up to 16. A two-stage ring overlaps the split of one
// k-block with the products of the other; the producer warps then read the
// accumulator back (tcgen05.ld) and apply the phase's epilogue. Waits are
// bounded; a CTA that gives up records a code in *err and unwinds.
constexpr int kTcM = 128, kTcN = 128, kTcK = 64;   // tile, k-block of bf16 (one 128-byte row)
constexpr int kTcStages = 1;                        // one stage: two CTAs share an SM and overlap
constexpr int kTcProd = 8;                          // producer (and epilogue) warps
constexpr int kTcThreads = (kTcProd + 1) * 32;
constexpr int kTcPart = kTcM * kTcK * 2;            // one part of one operand tile: 16 KB
constexpr int kTcStage = 6 * kTcPart;               // A h m l, B h m l
constexpr int kTcSmem = kTcStages * kTcStage + 1024 + 256;

// Eight consecutive k of one row of an operand tile, split into three parts
// and stored at 16-byte chunk `ch` of row `row` (128-byte swizzle).
__device__ __forceinline__ uint32_t bf2_bits(__nv_bfloat162 v) {
  return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ void split_store8(const float (&x)[8], unsigned char *part0, int row, int ch) {
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {  // two elements per packed conversion
    const __nv_bfloat162 h = __floats2bfloat162_rn(x[j], x[j + 1]);
    const float2 hf = __bfloat1622float2(h);
    const float r0 = x[j] - hf.x, r1 = x[j + 1] - hf.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(r0, r1);
    const float2 mf = __bfloat1622float2(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(r0 - mf.x, r1 - mf.y);
    w[0][j >> 1] = bf2_bits(h);
    w[1][j >> 1] = bf2_bits(m);
    w[2][j >> 1] = bf2_bits(l);
  }
  const int off = (row >> 3) * 1024 + (row & 7) * 128 + ((ch ^ (row & 7)) << 4);
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint4 *>(part0 + p * kTcPart + off) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

template <typename Item, typename Ops>
__global__ void __launch_bounds__(kTcThreads, 2)
    g_tc_kernel(const Item *__restrict__ items, const BPlan *__restrict__ plans,
                const int *__restrict__ tile_prefix, int batch, int phase, int *err) {
  using namespace tc;
  const int tile = blockIdx.x;
  int lo = 0, hi = batch - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_prefix[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  const Item it = items[lo];
  const BPlan pl = plans[lo];
  GOps<float> o;
  if (!Ops::pade(it, pl, phase, blockIdx.y, o)) return;  // uniform over the CTA
  const int n = it.n;
  const int tn = (n + kTcM - 1) / kTcM;
  const int local = tile - tile_prefix[lo];
  const int m0 = (local % tn) * kTcM, n0 = (local / tn) * kTcN;
  const int cols = min(kTcN, n - n0);
  const int Nt = (cols + 15) & ~15;
  const int nkb = (n + kTcK - 1) / kTcK;
  const int total = (o.A2 ? 2 : 1) * nkb;

  extern __shared__ __align__(1024) unsigned char tc_smem[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(tc_smem) + 1023) & ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(base + kTcStages * kTcStage);
  uint64_t *empty = full + kTcStages;
  uint64_t *acc_full = empty + kTcStages;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
  int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(&full[s], kTcProd * 32);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kTcProd) {
    tmem_alloc(tmem_slot, kTcN);
    fence_before();
  }
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < kTcProd) {
    // ---- producers: split k-block after k-block into the ring ----
    const int t = threadIdx.x;
    bool ok = true;
    for (int i = 0; i < total && ok; ++i) {
      const int s = i % kTcStages;
      const uint32_t ph = (uint32_t)((i / kTcStages) & 1);
      for (long long w = 0;; ++w) {
        if (mbar_try_wait(&empty[s], ph ^ 1u)) break;
        if (w >= kSpinLimit || ((w & 255) == 255 && *(volatile int *)abort_flag)) {
          record_error(err, 11);
          *(volatile int *)abort_flag = 1;
          ok = false;
          break;
        }
      }
      if (!ok) break;
      const bool second = i >= nkb;
      const float *Am = second ? o.A2 : o.A;
      const float *Bm = second ? o.B2 : o.B;
      const int lda = second ? o.lda2 : o.lda, ldb = second ? o.ldb2 : o.ldb;
      const int k0 = (second ? i - nkb : i) * kTcK;
      unsigned char *sa = base + s * kTcStage, *sb = sa + 3 * kTcPart;
      {  // A: four consecutive rows x one chunk of 8 k per thread; lanes along rows
        const int rq = t & 31, ch = t >> 5;
        const int gm = m0 + 4 * rq, kc = k0 + ch * 8;
        float x[4][8];
        const bool vec = gm + 3 < n && kc + 8 <= n && (lda & 3) == 0 &&
                         (reinterpret_cast<uintptr_t>(Am + gm) & 15) == 0;
        if (vec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 u = *reinterpret_cast<const float4 *>(Am + (std::size_t)(kc + j) * lda + gm);
            x[0][j] = u.x, x[1][j] = u.y, x[2][j] = u.z, x[3][j] = u.w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              x[r][j] = (gm + r < n && kc + j < n) ? Am[(std::size_t)(kc + j) * lda + gm + r] : 0.f;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) split_store8(x[r], sa, 4 * rq + r, ch);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // B: 128 columns x 8 chunks of 8 k; lanes along k
        const int id = t + q * (kTcProd * 32);
        const int ch = id & 7, row = id >> 3;
        const int gc = n0 + row, kc = k0 + ch * 8;
        float x[8];
        const float *src = Bm + (std::size_t)gc * ldb + kc;
        if (gc < n && kc + 8 <= n && ((reinterpret_cast<uintptr_t>(src) & 15) == 0)) {
          const float4 u = *reinterpret_cast<const float4 *>(src);
          const float4 v = *reinterpret_cast<const float4 *>(src + 4);
          x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) x[j] = (gc < n && kc + j < n) ? src[j] : 0.f;
        }
        split_store8(x, sb, row, ch);
      }
      // the generic-proxy stores become visible to the tensor cores' reads
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&full[s]);
    }
    // ---- epilogue ----
    bool got = false;
    for (long long w = 0; w < kSpinLimit; ++w) {
      if (mbar_try_wait(acc_full, 0)) {
        got = true;
        break;
      }
      if ((w & 255) == 255 && *(volatile int *)abort_flag) break;
    }
    if (!got && !*(volatile int *)abort_flag) record_error(err, 13);
    if (got && !*(volatile int *)abort_flag) {
      fence_after();
      const int q = warp & 3, half = warp >> 2;
      const int row = m0 + q * 32 + lane;
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 32) {
        const int cb = n0 + half * 64 + c0;
        if (cb >= n) break;  // warp-uniform
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * 64 + c0), v);
        if (row < n) {
#pragma unroll
          for (int j0 = 0; j0 < 32; j0 += 8) {  // old values of eight columns before their stores
            float old[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int c = cb + j0 + j;
              old[j] = (o.acc && c < n) ? o.C[(std::size_t)c * o.ldc + row] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int c = cb + j0 + j;
              if (c < n) {
                const float a = __uint_as_float(v[j0 + j]);
                o.C[(std::size_t)c * o.ldc + row] = o.neg ? old[j] - a : old[j] + a;
              }
            }
          }
        }
      }
    }
  } else if (lane == 0) {
    // ---- MMA issuer ----
    const uint32_t idesc = idesc_bf16_f32(kTcM, Nt);
    // (A part, B part) of the six products: l h, h l, m m, m h, h m, h h
    const int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
    bool ok = true;
    for (int i = 0; i < total; ++i) {
      const int s = i % kTcStages;
      const uint32_t ph = (uint32_t)((i / kTcStages) & 1);
      bool got = false;
      for (long long w = 0; w < kSpinLimit; ++w) {
        if (mbar_try_wait(&full[s], ph)) {
          got = true;
          break;
        }
        if ((w & 255) == 255 && *(volatile int *)abort_flag) break;
      }
      if (!got) {
        record_error(err, 12);
        *(volatile int *)abort_flag = 1;
        ok = false;
        break;
      }
      fence_after();
      const uint32_t sa = saddr(base + s * kTcStage), sb = sa + 3 * kTcPart;
#pragma unroll
      for (int tt = 0; tt < 6; ++tt)
#pragma unroll
        for (int k = 0; k < kTcK / 16; ++k)  // +32 bytes per 16-element k step inside the row
          mma_f16(tmem, smem_desc_sw128(sa + pa[tt] * kTcPart + k * 32),
                  smem_desc_sw128(sb + pb[tt] * kTcPart + k * 32), idesc, (i > 0 || tt > 0 || k > 0) ? 1u : 0u);
      mma_commit(&empty[s]);
    }
    (void)ok;
    mma_commit(acc_full);  // tracks every MMA above, on the abort path too
    if (!mbar_wait(acc_full, 0)) record_error(err, 14);
  }
  fence_before();
  __syncthreads();
  if (warp == kTcProd) {
    fence_after();
    tmem_dealloc(tmem, kTcN);
  }
}

inline int tiles128_of(int n) {
  const int t = (n + kTcM - 1) / kTcM;
  return t * t;
}

// The FP32 evaluation phases on the tensor cores (128-tile numbering).
template <typename Item, typename Ops>
cudaError_t launch_group_tc(cudaStream_t st, dim3 grid, const Item *items, const BPlan *plans,
                            const int *prefix128, int count, int phase, int *err) {
  static OncePerDevice once;
  auto kern = g_tc_kernel<Item, Ops>;
  const cudaError_t e = opt_in_smem(once, kern, kTcSmem);
  if (e != cudaSuccess) return e;
  kern<<<grid, kTcThreads, kTcSmem, st>>>(items, plans, prefix128, count, phase, err);
  return launched();
}

// Launch a grouped product phase on the engine of its element type: DMMA
// tiles for double, the SIMT kernel otherwise.
template <typename Item, typename U, typename Ops, bool kSquare>
cudaError_t launch_group(cudaStream_t st, dim3 grid, const Item *items, const BPlan *plans,
                         const int *prefix, int count, int phase, int k) {
  if constexpr (std::is_same<U, double>::value) {
    static OncePerDevice once;
    auto kern = g_dgemm_kernel<Item, Ops, kSquare>;
    const cudaError_t e = opt_in_smem(once, kern, kDSmem);
    if (e != cudaSuccess) return e;
    kern<<<grid, 128, kDSmem, st>>>(items, plans, prefix, count, phase, k);
  } else {
    g_gemm_kernel<Item, U, Ops, kSquare><<<grid, 256, 0, st>>>(items, plans, prefix, count, phase, k);
  }
  return launched();
}

// ---- LU with partial pivoting of q and the solve q R = p: one CTA per matrix
// Row loops update 8 columns at a time: eight independent loads are issued
// before the first store, so the L2 latency is paid once per eight elements.
constexpr int kBU = 8;

// CTAs per SM the LU kernel is compiled for: FP32 three 256-thread CTAs (80
// registers, a few spilled; three CTAs' shared memory fits; measured 2 %
// faster on the mixed tier than two at 128 registers, four no better); FP64
// as the solve kind says (Lu::kFp64Ctas): two
// CTAs (128 registers, a few spilled, and both CTAs' shared memory fit)
// measured faster for the expm solve, one (up to 255 registers) for the
// adjoint's, which spills more at 128.
template <typename T, int NT, typename Lu> struct BLuOcc {
  static constexpr int kMinBlocks = (sizeof(T) == 4 ? 3 : Lu::kFp64Ctas) * (256 / NT);
};

// D(r0 + i, c) -= sum_{j < jb} L(i, j) blk[j][c] for i < mrows, c in [c0, c0 + ncols),
// with L(i, j) = L[j * ldl + r0 + i] (column-major, global). All threads take
// part: 64 x (NT / 4) output blocks, thread (tr, tc) = (t % 16, t / 16) owns
// rows tr + 16 a and columns 4 tc + b (a, b < 4) of a block; L's 64 rows of a
// block are staged in shared memory. c0 is a multiple of 4 and blk rows are
// padded by at least 64 columns, so the 4-wide shared loads never leave their
// row; the padding also makes the row pitch 4 (mod 32) 4-byte words for float
// and 2 (mod 16) 8-byte words for double, so the row-block copies below hit
// 32 distinct banks.
template <typename T, int NT> constexpr int blk_ld() { return NT + (sizeof(T) == 4 ? 68 : 66); }

// Rows [k, k + jb) of the ncols columns of M (column-major, ld) outside
// [skip, skip + skipw) to blk[j][c] (kToShared) or back, c the column. Each
// warp instruction moves 8 consecutive rows of 4 columns: four contiguous
// 32-byte (float) or 64-byte (double) pieces, where a column per thread
// would touch 32 lines.
template <bool kToShared, typename T, int NT>
__device__ __forceinline__ void blk_rows(T *M, int ld, int k, int jb, int ncols, int skip, int skipw,
                                         T (*blk)[blk_ld<T, NT>()]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = 4 * ((ncols + 3) >> 2);
  for (int g = warp; g < groups; g += NT / 32) {
    const int j = (g & 3) * 8 + (lane & 7), ci = (g >> 2) * 4 + (lane >> 3);
    if (j < jb && ci < ncols) {
      const int c = ci < skip ? ci : ci + skipw;
      if (kToShared) blk[j][c] = M[(std::size_t)c * ld + k + j];
      else M[(std::size_t)c * ld + k + j] = blk[j][c];
    }
  }
}

// The jb x jb diagonal block of Q (ld n) at (k, k) to diag[row][column],
// consecutive threads reading down a column.
template <typename T, int NT>
__device__ __forceinline__ void stage_diag(const T *Q, int n, int k, int jb, T (*diag)[kBPanel + 1]) {
  for (int e = threadIdx.x; e < jb * jb; e += NT) {
    const int q = e / jb, j = e - q * jb;
    diag[j][q] = Q[(std::size_t)(k + q) * n + k + j];
  }
}

// Triangular solves of one right-hand-side column against the diagonal block
// in shared memory: unit lower (forward) and non-unit upper with the diagonal's
// reciprocals (backward). kFull: jb == kBPanel, so every bound is static.
template <typename T, bool kFull>
__device__ __forceinline__ void trsv_lower_unit(T (&x)[kBPanel], const T (*diag)[kBPanel + 1], int jb) {
#pragma unroll
  for (int j = 1; j < kBPanel; ++j)
#pragma unroll
    for (int q = 0; q < j; ++q)
      if (kFull || j < jb) x[j] = sub(x[j], mul(diag[j][q], x[q]));
}

template <typename T, bool kFull>
__device__ __forceinline__ void trsv_upper(T (&x)[kBPanel], const T (*diag)[kBPanel + 1], const T *rdiag,
                                           int jb) {
#pragma unroll
  for (int j = kBPanel - 1; j >= 0; --j) {
    if (kFull || j < jb) {
#pragma unroll
      for (int q = j + 1; q < kBPanel; ++q)
        if (kFull || q < jb) x[j] = sub(x[j], mul(diag[j][q], x[q]));
      x[j] = mul(x[j], rdiag[j]);
    }
  }
}

template <typename T, int NT>
__device__ void cta_update(T *__restrict__ D, int ldd, int r0, int mrows, int c0, int ncols,
                           const T *__restrict__ L, int ldl, int jb,
                           const T (*__restrict__ blk)[blk_ld<T, NT>()], T (*__restrict__ Ls)[64]) {
  constexpr int CB = NT / 4;  // columns per block
  const int t = threadIdx.x, tr = t & 15, tc = t >> 4;
  for (int rb = 0; rb < mrows; rb += 64) {
    __syncthreads();  // Ls is rewritten
    for (int e = t; e < 64 * kBPanel; e += NT) {
      const int i = e & 63, j = e >> 6;
      Ls[j][i] = (j < jb && rb + i < mrows) ? L[(std::size_t)j * ldl + r0 + rb + i] : elem<T>::zero();
    }
    __syncthreads();
    for (int cb = 0; cb < ncols; cb += CB) {
      T acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = elem<T>::zero();
      const int cc = c0 + cb + 4 * tc;
      // the block's old values are requested before the k loop, so their
      // latency overlaps the products
      T old[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = rb + tr + 16 * a, c = cc + b;
          old[a][b] = (i < mrows && c < c0 + ncols) ? D[(std::size_t)c * ldd + r0 + i] : elem<T>::zero();
        }
#pragma unroll 4
      for (int j = 0; j < jb; ++j) {
        T av[4], bv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) av[a] = Ls[j][tr + 16 * a];
        lds4(&blk[j][cc], bv);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = fmac(av[a], bv[b], acc[a][b]);
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = rb + tr + 16 * a, c = cc + b;
          if (i < mrows && c < c0 + ncols) D[(std::size_t)c * ldd + r0 + i] = sub(old[a][b], acc[a][b]);
        }
    }
  }
  __syncthreads();
}

// What the LU kernel factors and solves for one matrix: q (factored in place,
// ld n), the right-hand side B (ld n), the solution D (ldd), where the row
// permutation is kept for a later solve with the same factors (may be null),
// and the matrix's index in the caller's batch (info).
template <typename T>
struct LuOps {
  T *Q;
  const T *B;
  T *D;
  int ldd;
  int *perm;
  int id;
};

// expm: factor q = V, solve for the quotient from p (in P0) into the output
// (s = 0) or into X (s > 0, squared afterwards)
struct ExpmLu {
  static constexpr int kFp64Ctas = 2;
  template <typename T, typename Wd>
  static __device__ __forceinline__ LuOps<T> ops(const BItem<T, Wd> &it, const BPlan &pl, int) {
    return LuOps<T>{it.V, it.P0, pl.s > 0 ? it.X : it.E, pl.s > 0 ? it.n : it.lde, nullptr, it.id};
  }
};

// kFactor: LU with partial pivoting of Q, then the solve; otherwise the solve
// alone with factors and permutation from an earlier kFactor launch.
// kLongFirst: the matrices, sorted by ascending n, from the last on.
template <typename Item, typename T, typename Lu, bool kFactor, int NT, bool kLongFirst>
__global__ void __launch_bounds__(NT, BLuOcc<T, NT, Lu>::kMinBlocks)
    g_lu_kernel(const Item *__restrict__ items, const BPlan *__restrict__ plans, int *__restrict__ info,
                int mode) {
  using R = typename elem<T>::real;
  const int item = kLongFirst ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const Item it = items[item];
  const BPlan pl = plans[item];
  const int n = it.n;
  const LuOps<T> lo = Lu::ops(it, pl, mode);
  T *Q = lo.Q;
  const T *B = lo.B;
  T *D = lo.D;
  const int ldd = lo.ldd;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

  // dynamic: blk[kBPanel][NT + 64] (per-column staging, U12 rows, solved
  // right-hand-side block rows), Ls[kBPanel][64] (staged L rows of the block
  // updates), then diag[kBPanel][kBPanel + 1]
  extern __shared__ __align__(16) unsigned char b_smem[];
  constexpr int LD = blk_ld<T, NT>();
  auto blk = reinterpret_cast<T(*)[LD]>(b_smem);
  auto Ls = reinterpret_cast<T(*)[64]>(b_smem + sizeof(T) * kBPanel * LD);
  auto diag = reinterpret_cast<T(*)[kBPanel + 1]>(b_smem + sizeof(T) * kBPanel * (LD + 64));
  // per pivot step, alternating: slot 0 the pivot row, slot 1 row a before
  // the exchange; the pivot's reciprocal
  __shared__ __align__(16) T wrow[2][2][kBPanel];
  __shared__ T wrcp[2][1];
  __shared__ T rdiag[kBPanel];     // reciprocals of U's diagonal block
  __shared__ int perm[NT];  // P: row i of P q is row perm[i] of q
  __shared__ int pos[NT];   // panel-local composite of the swaps
  __shared__ int piv[kBPanel];
  __shared__ unsigned long long red_key[2][NT / 32];
  __shared__ int red_idx[2][NT / 32];
  __shared__ int first_zero;

  if (t < n) perm[t] = kFactor ? t : lo.perm[t];
  if (t == 0) first_zero = 0;
  const double sfmin = sizeof(R) == 4 ? (double)FLT_MIN : DBL_MIN;

  T r[kBPanel];
  for (int k = 0; k < (kFactor ? n : 0); k += kBPanel) {
    const int jb = min(kBPanel, n - k);
    const bool mine = t >= k && t < n;
#pragma unroll
    for (int j = 0; j < kBPanel; ++j)
      r[j] = (mine && j < jb) ? Q[(std::size_t)(k + j) * n + t] : elem<T>::zero();
    if (t < n) pos[t] = t;
    __syncthreads();
    // One pivot column per step. Each row's registers rotate one place left
    // after every step, so the pivot column is always r[0] and the rolled loop
    // has static register indices; finished columns ride at the back (still
    // exchanged with their row) and the update is masked to the unfinished
    // positions. After kBPanel steps (idle ones past jb) the row is back in
    // column order. Two barriers per step: the CTA argmax (warp winners form
    // their row's reciprocal meanwhile), then the pivot row (slot 0) and row a
    // (slot kX) are published. With one row per thread this measured faster
    // than publishing every warp winner's row before a single barrier.
    constexpr int kX = 1;  // the slot of row a
#pragma unroll 1
    for (int j = 0; j < kBPanel; ++j) {
      if (j < jb) {
        const int a = k + j, buf = j & 1;
        // pivot: largest |Re| + |Im| among rows >= a, first index on ties
        const ArgMax wa = warp_argmax(argmax_key(abs1(r[0]), t, mine && t >= a));
        cta_argmax_publish(wa, red_key[buf], red_idx[buf]);
        T myrcp = elem<T>::one();
        if (t == wa.idx && !is_zero(r[0])) myrcp = divide(elem<T>::one(), r[0]);
        __syncthreads();
        const ArgMax am = cta_argmax_collect(red_key[buf], red_idx[buf]);
        const double bv = __longlong_as_double((long long)am.key);
        int p = am.idx;
        const bool forced = p >= n;  // no comparable candidate (NaN column): keep row a
        if (forced) p = a;
        if (t == a) {
#pragma unroll
          for (int c = 0; c < kBPanel; ++c) wrow[buf][kX][c] = r[c];
        }
        if (t == p) {
#pragma unroll
          for (int c = 0; c < kBPanel; ++c) wrow[buf][0][c] = r[c];
          wrcp[buf][0] = myrcp;
        }
        const T *prow = wrow[buf][0];
        if (t == 0) {
          piv[j] = p;
          if (p != a) {
            const int tp = perm[a];
            perm[a] = perm[p];
            perm[p] = tp;
            const int tq = pos[a];
            pos[a] = pos[p];
            pos[p] = tq;
          }
          if (!(bv > 0.0) && first_zero == 0) first_zero = a + 1;
        }
        __syncthreads();
        if (p != a) {
          if (t == a) {
#pragma unroll
            for (int c = 0; c < kBPanel; c += 4) {
              T u[4];
              lds4(&prow[c], u);
#pragma unroll
              for (int i = 0; i < 4; ++i) r[c + i] = u[i];
            }
          } else if (t == p) {
#pragma unroll
            for (int c = 0; c < kBPanel; c += 4) {
              T u[4];
              lds4(&wrow[buf][kX][c], u);
#pragma unroll
              for (int i = 0; i < 4; ++i) r[c + i] = u[i];
            }
          }
        }
        const T pv = prow[0];
        if (mine && t > a && !is_zero(pv)) {
          T l = r[0];
          l = (!forced && abs1(pv) >= sfmin) ? mul(l, wrcp[buf][0]) : divide(l, pv);
          const int lim = jb - j;  // positions 1 .. lim-1 hold unfinished columns
#pragma unroll
          for (int c = 0; c < kBPanel; c += 4) {
            T u[4];
            lds4(&prow[c], u);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c + i > 0 && c + i < lim) r[c + i] = sub(r[c + i], mul(l, u[i]));
          }
          r[0] = l;
        }
      }
      const T t0 = r[0];
#pragma unroll
      for (int c = 0; c + 1 < kBPanel; ++c) r[c] = r[c + 1];
      r[kBPanel - 1] = t0;
    }
    // panel back to memory; L11 to shared memory
    if (mine) {
#pragma unroll
      for (int j = 0; j < kBPanel; ++j)
        if (j < jb) Q[(std::size_t)(k + j) * n + t] = r[j];
    }
    if (t >= k && t < k + jb) {
#pragma unroll
      for (int j = 0; j < kBPanel; ++j)
        if (j < jb) diag[t - k][j] = r[j];
    }
    // columns outside the panel: the old top block to shared memory
    blk_rows<true, T, NT>(Q, n, k, jb, n - jb, k, jb, blk);
    __syncthreads();
    // apply the panel's swaps (rows >= k + jb only ever receive rows of the
    // top block [k, k + jb)), then, right of the panel, solve the top block
    // with the unit-lower L11; the new top block goes back through blk
    if (t < n - jb) {
      const int c = t < k ? t : t + jb;
      T *col = Q + (std::size_t)c * n;
      T x[kBPanel];
#pragma unroll
      for (int j = 0; j < kBPanel; ++j) {
        x[j] = elem<T>::zero();
        if (j < jb) {
          const int src = pos[k + j];
          x[j] = src >= k + jb ? col[src] : blk[src - k][c];
        }
      }
#pragma unroll
      for (int j = 0; j < kBPanel; ++j) {
        if (j < jb) {
          const int d = piv[j];
          if (d >= k + jb) col[d] = blk[pos[d] - k][c];
        }
      }
      if (c >= k + jb) {
        if (jb == kBPanel) trsv_lower_unit<T, true>(x, diag, jb);
        else trsv_lower_unit<T, false>(x, diag, jb);
      }
#pragma unroll
      for (int j = 0; j < kBPanel; ++j)
        if (j < jb) blk[j][c] = x[j];
    }
    __syncthreads();
    blk_rows<false, T, NT>(Q, n, k, jb, n - jb, k, jb, blk);
    // trailing update A22 -= L21 U12 by the whole CTA (its first barrier
    // orders the copy above before blk is rewritten)
    cta_update<T, NT>(Q, n, k + jb, n - k - jb, k + jb, n - k - jb, Q + (std::size_t)k * n, n, jb, blk, Ls);
  }
  if (kFactor) {
    if (t == 0) {
      info[2 * lo.id] = first_zero;
      info[2 * lo.id + 1] = 0;
    }
    __syncthreads();
    if (lo.perm != nullptr && t < n) lo.perm[t] = perm[t];
  }
  __syncthreads();

  // ---- solve q R = p:  R = U^-1 L^-1 (P p) -------------------------------
  if (t < n) {
    const int src = perm[t];
    for (int c = 0; c < n; c += kBU) {
      T v[kBU];
#pragma unroll
      for (int u = 0; u < kBU; ++u) v[u] = c + u < n ? B[(std::size_t)(c + u) * n + src] : elem<T>::zero();
#pragma unroll
      for (int u = 0; u < kBU; ++u)
        if (c + u < n) D[(std::size_t)(c + u) * ldd + t] = v[u];
    }
  }
  __syncthreads();
  // forward, unit lower
  for (int k = 0; k < n; k += kBPanel) {
    const int jb = min(kBPanel, n - k);
    stage_diag<T, NT>(Q, n, k, jb, diag);
    blk_rows<true, T, NT>(D, ldd, k, jb, n, n, 0, blk);
    __syncthreads();
    if (t < n) {
      T x[kBPanel];
#pragma unroll
      for (int j = 0; j < kBPanel; ++j) x[j] = j < jb ? blk[j][t] : elem<T>::zero();
      if (jb == kBPanel) trsv_lower_unit<T, true>(x, diag, jb);
      else trsv_lower_unit<T, false>(x, diag, jb);
#pragma unroll
      for (int j = 0; j < kBPanel; ++j)
        if (j < jb) blk[j][t] = x[j];
    }
    __syncthreads();
    blk_rows<false, T, NT>(D, ldd, k, jb, n, n, 0, blk);
    cta_update<T, NT>(D, ldd, k + jb, n - k - jb, 0, n, Q + (std::size_t)k * n, n, jb, blk, Ls);
  }
  // backward, non-unit upper
  for (int k = ((n - 1) / kBPanel) * kBPanel; k >= 0; k -= kBPanel) {
    const int jb = min(kBPanel, n - k);
    stage_diag<T, NT>(Q, n, k, jb, diag);
    blk_rows<true, T, NT>(D, ldd, k, jb, n, n, 0, blk);
    __syncthreads();
    if (t < jb) rdiag[t] = divide(elem<T>::one(), diag[t][t]);
    __syncthreads();
    if (t < n) {
      T x[kBPanel];
#pragma unroll
      for (int j = 0; j < kBPanel; ++j) x[j] = j < jb ? blk[j][t] : elem<T>::zero();
      if (jb == kBPanel) trsv_upper<T, true>(x, diag, rdiag, jb);
      else trsv_upper<T, false>(x, diag, rdiag, jb);
#pragma unroll
      for (int j = 0; j < kBPanel; ++j)
        if (j < jb) blk[j][t] = x[j];
    }
    __syncthreads();
    blk_rows<false, T, NT>(D, ldd, k, jb, n, n, 0, blk);
    cta_update<T, NT>(D, ldd, 0, k, 0, n, Q + (std::size_t)k * n, n, jb, blk, Ls);
  }
}

template <typename T, int NT> constexpr std::size_t lu_smem_bytes() {
  return sizeof(T) * (kBPanel * (blk_ld<T, NT>() + 64) + kBPanel * (kBPanel + 1));
}

// The LU kernel over a batch sorted by n (ascending), one launch per run of
// matrices that share a CTA size: by default 64-thread CTAs for n <= 64, 128
// for n <= 128, 256 above (small matrices pack more CTAs per SM); a schedule
// (lu_threads[ceil(n / 16)], each >= n) may choose per size bucket.
// A batch of few matrices (lu_fork below) of more than one class leaves SMs idle at
// the end of every launch, and the launches are of unlike length: there the classes
// run beside one another, the longest CTAs first, the longest class on st and the
// others on the forked streams.
template <typename Item, typename T, typename Lu, bool kFactor>
cudaError_t launch_lu(cudaStream_t st, const Item *items, const BPlan *plans, int *info, int mode,
                      const std::vector<int> &ns, LuFork *fork, const int *lu_threads = nullptr) {
  const int count = (int)ns.size();
  auto threads_of = [&](int n) {
    const int d = n <= 64 ? 64 : n <= 128 ? 128 : 256;
    if (lu_threads == nullptr) return d;
    const int t = lu_threads[(n + 15) / 16];
    return (t == 64 || t == 128 || t == 256) && t >= n ? t : d;
  };
  auto one = [&](auto nt_tag, auto long_first, cudaStream_t on, int from, int to) -> cudaError_t {
    constexpr int NT = decltype(nt_tag)::value;
    auto kern = g_lu_kernel<Item, T, Lu, kFactor, NT, decltype(long_first)::value>;
    constexpr std::size_t smem = lu_smem_bytes<T, NT>();
    static OncePerDevice once;
    // the largest shared-memory carveout, so the CTAs the registers allow fit
    const cudaError_t e = opt_in_smem(once, kern, smem, 100);
    if (e != cudaSuccess) return e;
    kern<<<to - from, NT, smem, on>>>(items + from, plans + from, info, mode);
    return launched();
  };
  auto run = [&](auto long_first, cudaStream_t on, int from, int to) -> cudaError_t {
    const int nt = threads_of(ns[from]);
    return nt == 64    ? one(std::integral_constant<int, 64>{}, long_first, on, from, to)
           : nt == 128 ? one(std::integral_constant<int, 128>{}, long_first, on, from, to)
                       : one(std::integral_constant<int, 256>{}, long_first, on, from, to);
  };
  cudaError_t e = cudaSuccess;
  const bool classes = std::any_of(ns.begin(), ns.end(), [&](int n) { return threads_of(n) != threads_of(ns[0]); });
  if (fork == nullptr || !classes) {
    for (int from = 0, to; from < count && e == cudaSuccess; from = to) {
      for (to = from + 1; to < count && threads_of(ns[to]) == threads_of(ns[from]);) ++to;
      e = run(std::false_type{}, st, from, to);
    }
    return e;
  }
  if ((e = fork->create()) != cudaSuccess || (e = cudaEventRecord(fork->begin, st)) != cudaSuccess) return e;
  int used = 0;  // forked streams
  for (int to = count, from, c = 0; to > 0 && e == cudaSuccess; to = from, ++c) {
    for (from = to - 1; from > 0 && threads_of(ns[from - 1]) == threads_of(ns[to - 1]);) --from;
    const int k = (c - 1) % LuFork::kStreams;
    if (c > 0 && c <= LuFork::kStreams) {
      if ((e = cudaStreamWaitEvent(fork->s[k], fork->begin, 0)) != cudaSuccess) break;
      used = c;
    }
    e = run(std::true_type{}, c == 0 ? st : fork->s[k], from, to);
  }
  for (int k = 0; k < used; ++k) {  // after an error too: the call's stream stays behind what was launched
    cudaError_t j = cudaEventRecord(fork->end[k], fork->s[k]);
    if (j == cudaSuccess) j = cudaStreamWaitEvent(st, fork->end[k], 0);
    if (e == cudaSuccess) e = j;
  }
  return e;
}

// ---- precision conversion between the caller's buffers and FP64 copies ----
struct BConv {
  const void *src;
  void *dst;
  int n, lds, ldd, pad;
};

template <typename Ti, typename To>
__global__ void __launch_bounds__(256) b_conv_kernel(const BConv *__restrict__ conv) {
  const BConv cv = conv[blockIdx.x];
  const Ti *src = static_cast<const Ti *>(cv.src);
  To *dst = static_cast<To *>(cv.dst);
  const int n = cv.n, nn = n * n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    const int c = e / n, r = e - c * n;
    dst[(std::size_t)c * cv.ldd + r] = convert_elem<To>(src[(std::size_t)c * cv.lds + r]);
  }
}

// ---- host side -------------------------------------------------------------
// Workspace: [items (compute type T) | items (FP64) | plans x2 | tile prefixes
// x2 | norms | conversion tables x2 | one slab per matrix]. A matrix's slab is
// large enough for whichever precision its plan sends it to: the single tier
// keeps matrices with s = 0 in FP32 and evaluates matrices with s > 0 wholly
// in FP64 (their FP32 Pade quotient would carry ~1e-7 relative error into s
// squarings, each of which doubles it), from an FP64 copy of the input into
// an FP64 result that is rounded once into the caller's output.
template <typename T>
struct BLayout {
  using Hi = typename Wide<T>::type;
  static constexpr bool kSplit = !std::is_same<T, Hi>::value;
  std::size_t items_lo = 0, items_hi = 0, plans_lo = 0, plans_hi = 0, prefix_lo = 0, prefix_hi = 0,
              prefix128_lo = 0, err = 0, norms = 0, conv_in = 0, conv_out = 0, total = 0;
  std::vector<std::size_t> slab;
  template <typename C> static std::size_t slab_of(int n) {
    using W = typename Wide<C>::type;
    const std::size_t nn = (std::size_t)n * n;
    return 8 * align_up(nn * sizeof(C), 256) + 2 * align_up(nn * sizeof(W), 256);
  }
  static std::size_t slab_bytes(int n) {
    if (!kSplit) return slab_of<T>(n);
    const std::size_t nn = (std::size_t)n * n;
    return std::max(slab_of<T>(n), slab_of<Hi>(n) + 2 * align_up(nn * sizeof(Hi), 256));
  }
  void plan(int batch, const int *h_n) {
    Layout L(nullptr);
    items_lo = L.used;  L.take<BItem<T, Hi>>(batch);
    items_hi = L.used;  L.take<BItem<Hi, Hi>>(kSplit ? batch : 0);
    plans_lo = L.used;  L.take<BPlan>(batch);
    plans_hi = L.used;  L.take<BPlan>(kSplit ? batch : 0);
    prefix_lo = L.used; L.take<int>(batch + 1);
    prefix_hi = L.used; L.take<int>(kSplit ? batch + 1 : 0);
    prefix128_lo = L.used; L.take<int>(batch + 1);
    err = L.used;       L.take<int>(1);
    norms = L.used;     L.take<double>(batch);
    conv_in = L.used;   L.take<BConv>(kSplit ? batch : 0);
    conv_out = L.used;  L.take<BConv>(kSplit ? batch : 0);
    slab.resize(batch);
    std::size_t at = L.used;
    for (int i = 0; i < batch; ++i) {
      slab[i] = at;
      at += slab_bytes(h_n[i]);
    }
    total = at;
  }
};

bool g_pade_uploaded[64] = {};

cudaError_t upload_pade_table(int device) {
  if (device >= 0 && device < 64 && g_pade_uploaded[device]) return cudaSuccess;
  double tab[5][14] = {};
  const int ms[5] = {3, 5, 7, 9, 13};
  for (int k = 0; k < 5; ++k)
    for (int i = 0; i <= ms[k]; ++i) tab[k][i] = pade_coeffs(ms[k])[i];
  const cudaError_t e = cudaMemcpyToSymbol(c_pade, tab, sizeof(tab));
  if (e == cudaSuccess && device >= 0 && device < 64) g_pade_uploaded[device] = true;
  return e;
}

// The slab buffers of one matrix in compute type C.
template <typename C>
void carve_item(BItem<C, typename Wide<C>::type> &it, char *slab, int n) {
  using W = typename Wide<C>::type;
  const std::size_t nn = (std::size_t)n * n;
  Layout L(slab);
  it.X = L.take<C>(nn);
  it.P0 = L.take<C>(nn);
  it.P1 = L.take<C>(nn);
  it.P2 = L.take<C>(nn);
  it.P3 = L.take<C>(nn);
  it.Tt = L.take<C>(nn);
  it.V = L.take<C>(nn);
  it.W = L.take<C>(nn);
  it.wa = L.take<W>(nn);
  it.wb = L.take<W>(nn);
  it.n = n;
}

// Every phase over `count` matrices whose descriptors, plans and tile prefix
// sums are on the device.
// With kernel timing on (calamanSetKernelTiming), CUDA events bracket every
// grouped-GEMM launch, recorded with the launch's algorithmic flops.
template <typename F>
cudaError_t timed_group(cudaStream_t s, double flops, F &&run) {
  KernelTimer *t = tl_timer;
  if (t == nullptr || flops <= 0.0) return run();
  cudaEvent_t a = t->take(), b = t->take();
  if (a == nullptr || b == nullptr) return run();
  cudaEventRecord(a, s);
  const cudaError_t e = run();
  cudaEventRecord(b, s);
  t->starts.push_back(a);
  t->stops.push_back(b);
  t->flops.push_back(flops);
  return e;
}

// Algorithmic flops of a grouped-GEMM phase (k: the squaring index).
double phase_flops(const std::vector<int> &ns, const std::vector<BPlan> &pls, int phase, int k) {
  double f = 0.0;
  for (std::size_t i = 0; i < ns.size(); ++i) {
    const double cube = 2.0 * ns[i] * (double)ns[i] * ns[i];
    const BPlan &p = pls[i];
    switch (phase) {
    case kPhA2: case kPhU: f += cube; break;
    case kPhA4: f += p.np >= 2 ? cube : 0.0; break;
    case kPhA6: f += p.np >= 3 ? cube : 0.0; break;
    case kPhA8: f += p.np >= 4 ? cube : 0.0; break;
    case kPhM13: f += p.m == 13 ? 2.0 * cube : 0.0; break;
    case kPhSq: f += p.s >= k ? cube : 0.0; break;
    default: break;
    }
  }
  return f;
}

// FP32 items [tc_first, count) run their products on the tensor cores, with
// the 128-tile numbering d_prefix128 of that range (tiles128 tiles); items
// [0, tc_first) on the SIMT kernel with the 64-tile numbering d_prefix. The
// FP64 items' products stay on DMMA tiles. lu_threads: the LU's schedule.
template <typename C>
cudaError_t run_phases(cudaStream_t st, const BItem<C, typename Wide<C>::type> *d_items,
                       const BPlan *d_plans, const int *d_prefix, int count, int tiles, int max_n,
                       int max_s, int *d_info, const std::vector<int> &ns,
                       const std::vector<BPlan> &pls, const int *d_prefix128 = nullptr, int tiles128 = 0,
                       int *d_err = nullptr, int tc_first = 0, int tiles_simt = 0,
                       LuFork *fork = nullptr, const int *lu_threads = nullptr) {
  using W = typename Wide<C>::type;
  cudaError_t e;
  const dim3 ew((unsigned)count, (unsigned)((max_n * max_n + kEwChunk - 1) / kEwChunk));
  auto gemm = [&](int phase, int ysub) -> cudaError_t {
    return timed_group(st, phase_flops(ns, pls, phase, 0), [&] {
      if constexpr (std::is_same<C, float>::value) {
        if (d_prefix128) {
          cudaError_t e2 = cudaSuccess;
          if (tc_first > 0 && tiles_simt > 0)
            e2 = launch_group<BItem<C, W>, C, ExpmOps, false>(st, dim3(tiles_simt, ysub), d_items, d_plans,
                                                              d_prefix, tc_first, phase, 0);
          if (e2 == cudaSuccess && tc_first < count && tiles128 > 0)
            e2 = launch_group_tc<BItem<C, W>, ExpmOps>(st, dim3(tiles128, ysub), d_items + tc_first,
                                                       d_plans + tc_first, d_prefix128, count - tc_first, phase,
                                                       d_err);
          return e2;
        }
      }
      return launch_group<BItem<C, W>, C, ExpmOps, false>(st, dim3(tiles, ysub), d_items, d_plans, d_prefix,
                                                           count, phase, 0);
    });
  };
  b_scale_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
  if ((e = launched()) != cudaSuccess) return e;
  for (int ph : {kPhA2, kPhA4, kPhA6, kPhA8})
    if ((e = gemm(ph, 1)) != cudaSuccess) return e;
  b_even_odd_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
  if ((e = launched()) != cudaSuccess) return e;
  if ((e = gemm(kPhM13, 2)) != cudaSuccess) return e;
  if ((e = gemm(kPhU, 1)) != cudaSuccess) return e;
  b_split_kernel<C, W><<<ew, 256, 0, st>>>(d_items);
  if ((e = launched()) != cudaSuccess) return e;
  if ((e = launch_lu<BItem<C, W>, C, ExpmLu, true>(st, d_items, d_plans, d_info, 0, ns, fork, lu_threads)) !=
      cudaSuccess)
    return e;
  if (max_s > 0) {
    b_widen_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
    if ((e = launched()) != cudaSuccess) return e;
    for (int k = 1; k <= max_s; ++k) {
      e = timed_group(st, phase_flops(ns, pls, kPhSq, k), [&] {
        return launch_group<BItem<C, W>, W, ExpmOps, true>(st, dim3(tiles, 1), d_items, d_plans, d_prefix,
                                                           count, kPhSq, k);
      });
      if (e != cudaSuccess) return e;
    }
    b_narrow_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
    if ((e = launched()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

inline int tiles_of(int n) {
  const int t = (n + kGTile - 1) / kGTile;
  return t * t;
}

// The handle's second stream for the FP64 matrices of a mixed batch (they
// share no buffer with the FP32 ones: one stream per precision pipeline keeps
// the tensor cores busy with FP32 products while the FP64 products and LUs
// run), created on first use with its fork and join events. side = nullptr:
// one stream (no handle, or kernel timing, or a batch of one precision).
cudaError_t side_stream(calamanHandle_t blas, bool want, cudaStream_t &side) {
  side = nullptr;
  if (!want || blas == nullptr || tl_timer != nullptr) return cudaSuccess;
  if (blas->side == nullptr) {
    cudaError_t e = cudaEventCreateWithFlags(&blas->side_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&blas->side_join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&blas->side, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
  }
  side = blas->side;
  return cudaSuccess;
}

// The forked streams of the LU's size classes: one set for the FP32 matrices, one
// for the FP64 ones, which may run at the same time. Calls of up to kForkItems
// matrices of both precisions, some four to sixteen CTAs per SM; null beyond, and
// without a handle to hold the streams. Plain against forked, us a call, n = 3 .. 200
// and norms 0.1 .. 100: float64 60 matrices 1351 -> 913, 500 2675 -> 2127, 1184 4448 ->
// 3888, 2048 7079 -> 6385; float32 (a mixed batch) 500 2335 -> 1793, 2048 4785 -> 4647,
// 3000 6757 -> 6804, 8192 18224 -> 18533: thousands fill every launch nearly to its end.
// (As programmatic dependent launches in one stream, whose CTAs wait at their end for
// the class before and hold their SM's slots meanwhile, 500 float64 took 2311, and the
// 8192 matrices in 16 sub-batches on 16 streams 233.9k expm/s from and to the host,
// against 266k plain and 274k so.)
constexpr int kForkItems = 16 * 148;
LuFork *lu_fork(calamanHandle_t blas, int fp64, int batch) {
  return blas != nullptr && batch <= kForkItems ? &blas->lu_fork[fp64] : nullptr;
}

// Fork (before) or join (after) the side stream around a call's launches.
cudaError_t side_fork(calamanHandle_t blas, cudaStream_t st, cudaStream_t side) {
  if (side == nullptr) return cudaSuccess;
  cudaError_t e = cudaEventRecord(blas->side_fork, st);
  return e == cudaSuccess ? cudaStreamWaitEvent(side, blas->side_fork, 0) : e;
}
cudaError_t side_join(calamanHandle_t blas, cudaStream_t st, cudaStream_t side) {
  if (side == nullptr) return cudaSuccess;
  cudaError_t e = cudaEventRecord(blas->side_join, side);
  return e == cudaSuccess ? cudaStreamWaitEvent(st, blas->side_join, 0) : e;
}

template <typename T>
calamanStatus_t batched_api(calamanHandle_t blas, calamanStream_t stream, int batch, const int *h_n,
                            const T *const *h_A, const int *h_lda, T *const *h_E, const int *h_lde,
                            void *work, std::size_t lwork, int *d_info, calamanExpmPlan_t *h_plans) {
  using R = typename elem<T>::real;
  using Hi = typename Wide<T>::type;
  using Lay = BLayout<T>;
  if (batch < 0) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (batch == 0) return ok_status();
  if (h_n == nullptr || h_A == nullptr || h_lda == nullptr || h_E == nullptr || h_lde == nullptr ||
      work == nullptr || d_info == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  for (int i = 0; i < batch; ++i) {
    if (h_n[i] < 1 || h_lda[i] < h_n[i] || h_lde[i] < h_n[i] || h_A[i] == nullptr || h_E[i] == nullptr)
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    if (h_n[i] > kBatchedMaxN) return blas_status(CALAMAN_STATUS_NOT_SUPPORTED);
  }
  Lay lay;
  lay.plan(batch, h_n);
  if (lwork < lay.total) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  PointerModeScope pm(blas);
  TimerScope ts(timer_of(blas));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int dev = 0;
  CLM_CUDA(cudaGetDevice(&dev));
  CLM_CUDA(upload_pade_table(dev));

  char *base = static_cast<char *>(work);
  auto *d_lo = reinterpret_cast<BItem<T, Hi> *>(base + lay.items_lo);
  auto *d_hi = reinterpret_cast<BItem<Hi, Hi> *>(base + lay.items_hi);
  auto *d_plo = reinterpret_cast<BPlan *>(base + lay.plans_lo);
  auto *d_phi = reinterpret_cast<BPlan *>(base + lay.plans_hi);
  auto *d_xlo = reinterpret_cast<int *>(base + lay.prefix_lo);
  auto *d_xhi = reinterpret_cast<int *>(base + lay.prefix_hi);
  auto *d_x128 = reinterpret_cast<int *>(base + lay.prefix128_lo);
  auto *d_err = reinterpret_cast<int *>(base + lay.err);
  auto *d_norms = reinterpret_cast<double *>(base + lay.norms);
  auto *d_cin = reinterpret_cast<BConv *>(base + lay.conv_in);
  auto *d_cout = reinterpret_cast<BConv *>(base + lay.conv_out);

  // 1. every 1-norm, one readback, every plan on the host
  std::vector<BItem<T, Hi>> lo(batch);
  for (int i = 0; i < batch; ++i) {
    BItem<T, Hi> &it = lo[i];
    carve_item<T>(it, base + lay.slab[i], h_n[i]);
    it.A = h_A[i];
    it.E = h_E[i];
    it.lda = h_lda[i];
    it.lde = h_lde[i];
    it.id = i;
  }
  // pageable sources: each copy returns once its data is staged
  CLM_CUDA(cudaMemcpyAsync(d_lo, lo.data(), sizeof(BItem<T, Hi>) * batch, cudaMemcpyHostToDevice, st));
  b_norm_kernel<BItem<T, Hi>><<<batch, 256, 0, st>>>(d_lo, d_norms);
  CLM_CUDA(launched());
  std::vector<double> norms(batch);
  CLM_CUDA(cudaMemcpyAsync(norms.data(), d_norms, sizeof(double) * batch, cudaMemcpyDeviceToHost, st));
  CLM_CUDA(cudaStreamSynchronize(st));
  std::vector<calamanExpmPlan_t> plans(batch);
  for (int i = 0; i < batch; ++i) {
    if (!std::isfinite(norms[i])) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    plans[i] = plan_for<R>((R)norms[i]);
  }
  if (h_plans)
    for (int i = 0; i < batch; ++i) h_plans[i] = plans[i];

  // 2. partition: the single tier sends s > 0 to FP64
  std::vector<BItem<T, Hi>> lo_items;
  std::vector<BItem<Hi, Hi>> hi_items;
  std::vector<BPlan> lo_plans, hi_plans;
  std::vector<int> lo_prefix(1, 0), hi_prefix(1, 0), lo_prefix128(1, 0), lo_n, hi_n;
  std::vector<BConv> cin, cout;
  int lo_max_n = 0, hi_max_n = 0, lo_max_s = 0, hi_max_s = 0;
  // matrices in ascending n: the LU runs one launch per size class
  std::vector<int> order(batch);
  for (int i = 0; i < batch; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return h_n[x] < h_n[y]; });
  for (int i : order) {
    const calamanExpmPlan_t &p = plans[i];
    const BPlan bp{p.m, p.s, pade_num_powers(p.m), 0};
    const int n = h_n[i];
    if (!Lay::kSplit || p.s == 0) {
      lo_items.push_back(lo[i]);
      lo_plans.push_back(bp);
      lo_prefix.push_back(lo_prefix.back() + tiles_of(n));
      lo_prefix128.push_back(lo_prefix128.back() + tiles128_of(n));
      lo_n.push_back(n);
      lo_max_n = std::max(lo_max_n, n);
      lo_max_s = std::max(lo_max_s, p.s);
    } else {
      BItem<Hi, Hi> it{};
      carve_item<Hi>(it, base + lay.slab[i], n);
      const std::size_t nn = (std::size_t)n * n;
      char *extra = base + lay.slab[i] + Lay::template slab_of<Hi>(n);
      Hi *a64 = reinterpret_cast<Hi *>(extra);
      Hi *e64 = reinterpret_cast<Hi *>(extra + align_up(nn * sizeof(Hi), 256));
      it.A = a64;
      it.lda = n;
      it.E = e64;
      it.lde = n;
      it.id = i;
      hi_items.push_back(it);
      hi_plans.push_back(bp);
      hi_prefix.push_back(hi_prefix.back() + tiles_of(n));
      hi_n.push_back(n);
      hi_max_n = std::max(hi_max_n, n);
      hi_max_s = std::max(hi_max_s, p.s);
      cin.push_back(BConv{h_A[i], a64, n, h_lda[i], n, 0});
      cout.push_back(BConv{e64, h_E[i], n, n, h_lde[i], 0});
    }
  }
  const int nlo = (int)lo_items.size(), nhi = (int)hi_items.size();
  const BatchedTuning tune = blas ? blas->tune : default_batched_tuning();
  const bool tc = std::is_same<T, float>::value;
  // the FP32 items from tc_first on take the tensor cores (items are in ascending n)
  int tc_first = 0;
  while (tc && tc_first < nlo && lo_n[tc_first] < tune.fp32_tc_min_n) ++tc_first;
  std::vector<int> tc_prefix(1, 0);
  for (int i = tc_first; i < nlo; ++i) tc_prefix.push_back(tc_prefix.back() + tiles128_of(lo_n[i]));
  // the call's tables (every call; the kernels read them from the workspace)
  if (nlo > 0) {
    CLM_CUDA(cudaMemcpyAsync(d_lo, lo_items.data(), sizeof(BItem<T, Hi>) * nlo, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_plo, lo_plans.data(), sizeof(BPlan) * nlo, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_xlo, lo_prefix.data(), sizeof(int) * (nlo + 1), cudaMemcpyHostToDevice, st));
    if (tc) {
      CLM_CUDA(cudaMemcpyAsync(d_x128, tc_prefix.data(), sizeof(int) * tc_prefix.size(), cudaMemcpyHostToDevice,
                               st));
      CLM_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    }
  }
  if (nhi > 0) {
    CLM_CUDA(cudaMemcpyAsync(d_hi, hi_items.data(), sizeof(BItem<Hi, Hi>) * nhi, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_phi, hi_plans.data(), sizeof(BPlan) * nhi, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_xhi, hi_prefix.data(), sizeof(int) * (nhi + 1), cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_cin, cin.data(), sizeof(BConv) * nhi, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_cout, cout.data(), sizeof(BConv) * nhi, cudaMemcpyHostToDevice, st));
  }
  // every kernel of the call; a mixed batch runs its FP64 matrices on the
  // handle's side stream, beside the FP32 ones
  cudaStream_t side = nullptr;
  CLM_CUDA(side_stream(blas, nlo > 0 && nhi > 0, side));
  auto launch_all = [&]() -> cudaError_t {
    cudaError_t e;
    if ((e = side_fork(blas, st, side)) != cudaSuccess) return e;
    if (nhi > 0) {
      cudaStream_t sh = side ? side : st;
      const dim3 ew((unsigned)nhi, (unsigned)((hi_max_n * hi_max_n + kEwChunk - 1) / kEwChunk));
      b_conv_kernel<T, Hi><<<ew, 256, 0, sh>>>(d_cin);
      if ((e = launched()) != cudaSuccess) return e;
      if ((e = run_phases<Hi>(sh, d_hi, d_phi, d_xhi, nhi, hi_prefix.back(), hi_max_n, hi_max_s, d_info, hi_n,
                              hi_plans, nullptr, 0, nullptr, 0, 0, lu_fork(blas, 1, batch), tune.lu_threads)) != cudaSuccess)
        return e;
      b_conv_kernel<Hi, T><<<ew, 256, 0, sh>>>(d_cout);
      if ((e = launched()) != cudaSuccess) return e;
    }
    if (nlo > 0 &&
        (e = run_phases<T>(st, d_lo, d_plo, d_xlo, nlo, lo_prefix.back(), lo_max_n, lo_max_s, d_info, lo_n,
                           lo_plans, tc ? d_x128 : nullptr, tc_prefix.back(), d_err, tc_first,
                           lo_prefix[tc_first], lu_fork(blas, 0, batch), tune.lu_threads)) != cudaSuccess)
      return e;
    return side_join(blas, st, side);
  };
  // Graph replay: the launches depend only on the call's configuration, so a
  // configuration seen twice in a row is captured once and replayed after.
  // Kernel timing (CUDA events per launch) runs the launches directly.
  // (the legacy default streams cannot be captured: those calls run directly)
  if (blas == nullptr || !blas->graphs || tl_timer != nullptr || st == nullptr || st == cudaStreamLegacy ||
      st == cudaStreamPerThread) {
    CLM_CUDA(launch_all());
    return ok_status();
  }
  unsigned long long key = 1469598103934665603ull;
  auto mix = [&key](unsigned long long v) { key = (key ^ v) * 1099511628211ull; };
  mix((unsigned long long)batch);
  mix(sizeof(T));
  mix(reinterpret_cast<std::uintptr_t>(work));
  mix((unsigned long long)lwork);
  mix(reinterpret_cast<std::uintptr_t>(d_info));
  mix(reinterpret_cast<std::uintptr_t>(st));
  mix((unsigned long long)tune.fp32_tc_min_n);
  for (int b = 0; b <= 16; ++b) mix((unsigned long long)tune.lu_threads[b]);
  for (int i = 0; i < batch; ++i) {
    mix((unsigned long long)h_n[i] | ((unsigned long long)plans[i].m << 32) |
        ((unsigned long long)plans[i].s << 48));
    mix(reinterpret_cast<std::uintptr_t>(h_A[i]));
    mix(reinterpret_cast<std::uintptr_t>(h_E[i]));
    mix((unsigned long long)h_lda[i] | ((unsigned long long)h_lde[i] << 32));
  }
  BatchedGraph &g = blas->graph[std::is_same<T, double>::value ? 1 : 0];
  if (g.exec != nullptr && g.key == key) {
    CLM_CUDA(cudaGraphLaunch(static_cast<cudaGraphExec_t>(g.exec), st));
    note_launch(g.launches);
    return ok_status();
  }
  if (g.seen != key) {  // first sighting: run directly
    g.seen = key;
    CLM_CUDA(launch_all());
    return ok_status();
  }
  const unsigned long long before = g_launch_count();
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    const cudaError_t el = launch_all();
    e = cudaStreamEndCapture(st, &graph);
    if (el != cudaSuccess) e = el;
  }
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e != cudaSuccess) {  // no graph for this handle: the launches run directly from now on
    cudaGetLastError();
    blas->graphs = 0;
    CLM_CUDA(launch_all());
    return ok_status();
  }
  if (g.exec) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(g.exec));
  g.exec = exec;
  g.key = key;
  g.launches = (unsigned)(g_launch_count() - before);
  CLM_CUDA(cudaGraphLaunch(exec, st));
  return ok_status();
}

template <typename T>
calamanStatus_t batched_bytes(int batch, const int *h_n, std::size_t *bytes) {
  if (batch < 0 || bytes == nullptr || (batch > 0 && h_n == nullptr))
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  for (int i = 0; i < batch; ++i) {
    if (h_n[i] < 1) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    if (h_n[i] > kBatchedMaxN) return blas_status(CALAMAN_STATUS_NOT_SUPPORTED);
  }
  BLayout<T> lay;
  lay.plan(batch, h_n);
  *bytes = batch > 0 ? lay.total : 0;
  return ok_status();
}

// ===========================================================================
// The adjoint of expm over a batch (new entry point, see vjp.cu for the
// method): per pair (A, G), X = 2^-s A^H, D = 2^-s G, and every evaluation
// phase carries its derivative -- grouped GEMM phases with two sub-problems
// (value, derivative), the quotient and its derivative through one LU, and
// (R, L) <- (R^2, R L + L R) squarings.
// ===========================================================================
template <typename T, typename Wd>
struct BVItem {
  const T *A, *G;  // inputs (lda, ldg)
  T *Dg, *E;       // outputs: gradient (ldd), expm(A) or null (lde)
  T *Xs, *Ds, *P0, *P1, *P2, *P3, *M0, *M1, *M2, *M3, *T1, *T2, *V, *W, *LV, *LW;
  Wd *wr, *wl, *wr2, *wl2;
  int *perm;
  int n, lda, ldg, ldd, lde, id;
};

constexpr int kPhRhs = 10;  // dp - dq R into T2

struct VjpOps {
  template <typename T, typename Wd>
  static __device__ __forceinline__ bool pade(const BVItem<T, Wd> &it, const BPlan &pl, int phase, int sub,
                                              GOps<T> &o) {
    const int n = it.n;
    o.lda = o.ldb = o.lda2 = o.ldb2 = o.ldc = n;
    auto two = [&](const T *a, const T *b, const T *a2, const T *b2, T *c) {
      o.A = a; o.B = b; o.A2 = a2; o.B2 = b2; o.C = c;
    };
    switch (phase) {
    case kPhA2:  // A2 = X X; dA2 = X D + D X
      if (sub == 0) two(it.Xs, it.Xs, nullptr, nullptr, it.P0);
      else two(it.Xs, it.Ds, it.Ds, it.Xs, it.M0);
      return sub < 2;
    case kPhA4:  // A4 = A2 A2; dA4 = A2 dA2 + dA2 A2
      if (sub == 0) two(it.P0, it.P0, nullptr, nullptr, it.P1);
      else two(it.P0, it.M0, it.M0, it.P0, it.M1);
      return sub < 2 && pl.np >= 2;
    case kPhA6:  // A6 = A4 A2; dA6 = dA4 A2 + A4 dA2
      if (sub == 0) two(it.P1, it.P0, nullptr, nullptr, it.P2);
      else two(it.M1, it.P0, it.P1, it.M0, it.M2);
      return sub < 2 && pl.np >= 3;
    case kPhA8:  // A8 = A4 A4; dA8 = A4 dA4 + dA4 A4
      if (sub == 0) two(it.P1, it.P1, nullptr, nullptr, it.P3);
      else two(it.P1, it.M1, it.M1, it.P1, it.M3);
      return sub < 2 && pl.np >= 4;
    case kPhM13:  // W += A6 W1, V += A6 Z1 and their derivatives
      o.acc = true;
      if (sub == 0) two(it.P2, it.T1, nullptr, nullptr, it.W);
      else if (sub == 1) two(it.P2, it.P3, nullptr, nullptr, it.V);
      else if (sub == 2) two(it.P2, it.T2, it.M2, it.T1, it.LW);
      else two(it.P2, it.M3, it.M2, it.P3, it.LV);
      return sub < 4 && pl.m == 13;
    case kPhU:  // U = X W; dU = X dW + D W
      if (sub == 0) two(it.Xs, it.W, nullptr, nullptr, it.T1);
      else two(it.Xs, it.LW, it.Ds, it.W, it.T2);
      return sub < 2;
    case kPhRhs:  // dp - dq R (R in P0)
      o.acc = true;
      o.neg = true;
      two(it.LV, it.P0, nullptr, nullptr, it.T2);
      return sub == 0;
    default:
      return false;
    }
  }
  // square k reads (wr, wl) for odd k, (wr2, wl2) for even k
  template <typename T, typename Wd>
  static __device__ __forceinline__ bool square(const BVItem<T, Wd> &it, const BPlan &pl, int sub, int k,
                                                GOps<Wd> &o) {
    const Wd *r = (k & 1) ? it.wr : it.wr2, *l = (k & 1) ? it.wl : it.wl2;
    Wd *r2 = (k & 1) ? it.wr2 : it.wr, *l2 = (k & 1) ? it.wl2 : it.wl;
    o.lda = o.ldb = o.lda2 = o.ldb2 = o.ldc = it.n;
    if (sub == 0) {
      o.A = r; o.B = r; o.C = r2;
    } else {
      o.A = r; o.B = l; o.A2 = l; o.B2 = r; o.C = l2;
    }
    return pl.s >= k && sub < 2;
  }
};

// mode 0: factor q = V, R = q^-1 p (p in T1) into P0; mode 1: dR = q^-1 T2 into M0
struct VjpLu {
  static constexpr int kFp64Ctas = 1;
  template <typename T, typename Wd>
  static __device__ __forceinline__ LuOps<T> ops(const BVItem<T, Wd> &it, const BPlan &, int mode) {
    return mode == 0 ? LuOps<T>{it.V, it.T1, it.P0, it.n, it.perm, it.id}
                     : LuOps<T>{it.V, it.T2, it.M0, it.n, it.perm, it.id};
  }
};

// Xs = 2^-s A^H (the transpose for real types), Ds = 2^-s G
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) v_prep_kernel(const BVItem<T, Wd> *__restrict__ items,
                                                     const BPlan *__restrict__ plans) {
  using R = typename elem<T>::real;
  const BVItem<T, Wd> it = items[blockIdx.x];
  const R f = (R)ldexp(1.0, -plans[blockIdx.x].s);
  const int n = it.n, nn = n * n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    const int c = e / n, r = e - c * n;
    it.Xs[e] = scale(conj_elem(it.A[(std::size_t)r * it.lda + c]), f);
    it.Ds[e] = scale(it.G[(std::size_t)c * it.ldg + r], f);
  }
}

// The Pade combinations of the powers (P) and of their derivatives (M). Four CTAs
// per SM (64 registers): at the 88 that the 16-byte pieces would take in float64,
// two CTAs had too few loads in flight (300 matrices of n = 99 61 -> 86 us, and 62 so;
// n = 100 64 -> 76, and 57 so).
template <typename T, typename Wd>
__global__ void __launch_bounds__(256, 4) v_even_odd_kernel(const BVItem<T, Wd> *__restrict__ items,
                                                            const BPlan *__restrict__ plans) {
  using R = typename elem<T>::real;
  const BVItem<T, Wd> it = items[blockIdx.x];
  const BPlan pl = plans[blockIdx.x];
  const double *b = c_pade[degree_slot(pl.m)];
  const int n = it.n;
  const T *P[4] = {it.P0, it.P1, it.P2, it.P3};
  const T *M[4] = {it.M0, it.M1, it.M2, it.M3};
  ew_for<T>(it.V, n * n, [&](auto piece, int e) {
    constexpr int W = decltype(piece)::value;
    if (pl.m != 13) {
      Pack<W, T> v, w, lv, lw;
#pragma unroll
      for (int i = 0; i < W; ++i) v.e[i] = w.e[i] = lv.e[i] = lw.e[i] = elem<T>::zero();
      for (int k = 0; k < pl.np; ++k) {
        const Pack<W, T> x = ew_load<W>(P[k] + e), y = ew_load<W>(M[k] + e);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          v.e[i] = rfma((R)b[2 * k + 2], x.e[i], v.e[i]);
          w.e[i] = rfma((R)b[2 * k + 3], x.e[i], w.e[i]);
          lv.e[i] = rfma((R)b[2 * k + 2], y.e[i], lv.e[i]);
          lw.e[i] = rfma((R)b[2 * k + 3], y.e[i], lw.e[i]);
        }
      }
      ew_diag<W>(e, n, [&](int i, bool diag) {
        if (diag) {
          v.e[i] = add_real(v.e[i], (R)b[0]);
          w.e[i] = add_real(w.e[i], (R)b[1]);
        }
      });
      ew_store<W>(it.V + e, v);
      ew_store<W>(it.W + e, w);
      ew_store<W>(it.LV + e, lv);
      ew_store<W>(it.LW + e, lw);
    } else {
      const Pack<W, T> x1 = ew_load<W>(it.P0 + e), x2 = ew_load<W>(it.P1 + e), x3 = ew_load<W>(it.P2 + e);
      const Pack<W, T> y1 = ew_load<W>(it.M0 + e), y2 = ew_load<W>(it.M1 + e), y3 = ew_load<W>(it.M2 + e);
      auto comb = [&](const Pack<W, T> &a1, const Pack<W, T> &a2, const Pack<W, T> &a3, int i1, int i2, int i3) {
        Pack<W, T> o;
#pragma unroll
        for (int i = 0; i < W; ++i)
          o.e[i] = rfma((R)b[i3], a3.e[i], rfma((R)b[i2], a2.e[i], scale(a1.e[i], (R)b[i1])));
        return o;
      };
      Pack<W, T> w = comb(x1, x2, x3, 3, 5, 7), v = comb(x1, x2, x3, 2, 4, 6);
      ew_diag<W>(e, n, [&](int i, bool diag) {
        if (diag) {
          w.e[i] = add_real(w.e[i], (R)b[1]);
          v.e[i] = add_real(v.e[i], (R)b[0]);
        }
      });
      ew_store<W>(it.T1 + e, comb(x1, x2, x3, 9, 11, 13));
      ew_store<W>(it.W + e, w);
      ew_store<W>(it.P3 + e, comb(x1, x2, x3, 8, 10, 12));
      ew_store<W>(it.V + e, v);
      ew_store<W>(it.T2 + e, comb(y1, y2, y3, 9, 11, 13));
      ew_store<W>(it.LW + e, comb(y1, y2, y3, 3, 5, 7));
      ew_store<W>(it.M3 + e, comb(y1, y2, y3, 8, 10, 12));
      ew_store<W>(it.LV + e, comb(y1, y2, y3, 2, 4, 6));
    }
  });
}

// p = V + U over T1, q = V - U over V; dp = dV + dU over T2, dq = dV - dU over LV
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) v_split_kernel(const BVItem<T, Wd> *__restrict__ items) {
  const BVItem<T, Wd> it = items[blockIdx.x];
  // one loop over both pairs: four loads in flight per step (a loop per pair: 300
  // float64 pairs of n = 99 54 us against 38, 131 of n = 51 16 against 11)
  ew_for<T>(it.V, it.n * it.n, [&](auto piece, int e) {
    constexpr int W = decltype(piece)::value;
    const Pack<W, T> u = ew_load<W>(it.T1 + e), v = ew_load<W>(it.V + e);
    const Pack<W, T> du = ew_load<W>(it.T2 + e), dv = ew_load<W>(it.LV + e);
    Pack<W, T> p, q, dp, dq;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      p.e[i] = add(v.e[i], u.e[i]);
      q.e[i] = sub(v.e[i], u.e[i]);
      dp.e[i] = add(dv.e[i], du.e[i]);
      dq.e[i] = sub(dv.e[i], du.e[i]);
    }
    ew_store<W>(it.T1 + e, p);
    ew_store<W>(it.V + e, q);
    ew_store<W>(it.T2 + e, dp);
    ew_store<W>(it.LV + e, dq);
  });
}

// s > 0: (wr, wl) = wide (R, dR)
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) v_widen_kernel(const BVItem<T, Wd> *__restrict__ items,
                                                      const BPlan *__restrict__ plans) {
  if (plans[blockIdx.x].s == 0) return;
  const BVItem<T, Wd> it = items[blockIdx.x];
  const int nn = it.n * it.n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    it.wr[e] = convert_elem<Wd>(it.P0[e]);
    it.wl[e] = convert_elem<Wd>(it.M0[e]);
  }
}

// outputs: the gradient (the last dR), and expm(A) = (the last R)^H if wanted
template <typename T, typename Wd>
__global__ void __launch_bounds__(256) v_out_kernel(const BVItem<T, Wd> *__restrict__ items,
                                                    const BPlan *__restrict__ plans) {
  const BVItem<T, Wd> it = items[blockIdx.x];
  const int s = plans[blockIdx.x].s;
  const int n = it.n, nn = n * n;
  const int end = min(nn, (int)(blockIdx.y + 1) * kEwChunk);
  for (int e = blockIdx.y * kEwChunk + threadIdx.x; e < end; e += blockDim.x) {
    const int c = e / n, r = e - c * n;
    T g, x;
    if (s == 0) {
      g = it.M0[e];
      x = it.P0[(std::size_t)r * n + c];
    } else {
      const Wd *lf = (s & 1) ? it.wl2 : it.wl, *rf = (s & 1) ? it.wr2 : it.wr;
      g = convert_elem<T>(lf[e]);
      x = convert_elem<T>(rf[(std::size_t)r * n + c]);
    }
    it.Dg[(std::size_t)c * it.ldd + r] = g;
    if (it.E) it.E[(std::size_t)c * it.lde + r] = conj_elem(x);
  }
}

template <typename C>
void carve_vitem(BVItem<C, typename Wide<C>::type> &it, char *slab, int n) {
  using W = typename Wide<C>::type;
  const std::size_t nn = (std::size_t)n * n;
  Layout L(slab);
  C **bufs[16] = {&it.Xs, &it.Ds, &it.P0, &it.P1, &it.P2, &it.P3, &it.M0, &it.M1,
                  &it.M2, &it.M3, &it.T1, &it.T2, &it.V,  &it.W,  &it.LV, &it.LW};
  for (C **b : bufs) *b = L.take<C>(nn);
  it.wr = L.take<W>(nn);
  it.wl = L.take<W>(nn);
  it.wr2 = L.take<W>(nn);
  it.wl2 = L.take<W>(nn);
  it.perm = L.take<int>(n);
  it.n = n;
}

template <typename C>
std::size_t vslab_of(int n) {
  using W = typename Wide<C>::type;
  const std::size_t nn = (std::size_t)n * n;
  return 16 * align_up(nn * sizeof(C), 256) + 4 * align_up(nn * sizeof(W), 256) + align_up(n * sizeof(int), 256);
}

template <typename C>
cudaError_t run_vjp_phases(cudaStream_t st, const BVItem<C, typename Wide<C>::type> *d_items,
                           const BPlan *d_plans, const int *d_prefix, int count, int tiles, int max_n,
                           int max_s, int *d_info, const std::vector<int> &ns,
                           const std::vector<BPlan> &pls, const int *d_prefix128 = nullptr, int tiles128 = 0,
                           int *d_err = nullptr, int tc_first = 0, int tiles_simt = 0, LuFork *fork = nullptr) {
  using W = typename Wide<C>::type;
  using Item = BVItem<C, W>;
  cudaError_t e;
  const dim3 ew((unsigned)count, (unsigned)((max_n * max_n + kEwChunk - 1) / kEwChunk));
  // flops of a phase: per matrix, the products its sub-problems carry
  auto vflops = [&](int phase, int k) {
    double f = 0.0;
    for (std::size_t i = 0; i < ns.size(); ++i) {
      const double cube = 2.0 * ns[i] * (double)ns[i] * ns[i];
      const BPlan &p = pls[i];
      switch (phase) {
      case kPhA2: case kPhU: f += 3 * cube; break;
      case kPhA4: f += p.np >= 2 ? 3 * cube : 0.0; break;
      case kPhA6: f += p.np >= 3 ? 3 * cube : 0.0; break;
      case kPhA8: f += p.np >= 4 ? 3 * cube : 0.0; break;
      case kPhM13: f += p.m == 13 ? 6 * cube : 0.0; break;
      case kPhRhs: f += cube; break;
      case kPhSq: f += p.s >= k ? 3 * cube : 0.0; break;
      default: break;
      }
    }
    return f;
  };
  auto gemm = [&](int phase, int ysub) -> cudaError_t {
    return timed_group(st, vflops(phase, 0), [&] {
      if constexpr (std::is_same<C, float>::value) {
        if (d_prefix128) {  // FP32 products of items [tc_first, count) on the tensor cores
          cudaError_t e2 = cudaSuccess;
          if (tc_first > 0 && tiles_simt > 0)
            e2 = launch_group<Item, C, VjpOps, false>(st, dim3(tiles_simt, ysub), d_items, d_plans, d_prefix,
                                                      tc_first, phase, 0);
          if (e2 == cudaSuccess && tc_first < count && tiles128 > 0)
            e2 = launch_group_tc<Item, VjpOps>(st, dim3(tiles128, ysub), d_items + tc_first, d_plans + tc_first,
                                               d_prefix128, count - tc_first, phase, d_err);
          return e2;
        }
      }
      return launch_group<Item, C, VjpOps, false>(st, dim3(tiles, ysub), d_items, d_plans, d_prefix, count,
                                                  phase, 0);
    });
  };

  v_prep_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
  if ((e = launched()) != cudaSuccess) return e;
  for (int ph : {kPhA2, kPhA4, kPhA6, kPhA8})
    if ((e = gemm(ph, 2)) != cudaSuccess) return e;
  v_even_odd_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
  if ((e = launched()) != cudaSuccess) return e;
  if ((e = gemm(kPhM13, 4)) != cudaSuccess) return e;
  if ((e = gemm(kPhU, 2)) != cudaSuccess) return e;
  v_split_kernel<C, W><<<ew, 256, 0, st>>>(d_items);
  if ((e = launched()) != cudaSuccess) return e;
  if ((e = launch_lu<Item, C, VjpLu, true>(st, d_items, d_plans, d_info, 0, ns, fork)) != cudaSuccess) return e;
  if ((e = gemm(kPhRhs, 1)) != cudaSuccess) return e;
  if ((e = launch_lu<Item, C, VjpLu, false>(st, d_items, d_plans, d_info, 1, ns, fork)) != cudaSuccess) return e;
  if (max_s > 0) {
    v_widen_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
    if ((e = launched()) != cudaSuccess) return e;
    for (int k = 1; k <= max_s; ++k) {
      e = timed_group(st, vflops(kPhSq, k), [&] {
        return launch_group<Item, W, VjpOps, true>(st, dim3(tiles, 2), d_items, d_plans, d_prefix, count,
                                                   kPhSq, k);
      });
      if (e != cudaSuccess) return e;
    }
  }
  v_out_kernel<C, W><<<ew, 256, 0, st>>>(d_items, d_plans);
  return launched();
}

// Workspace: [items (T) | items (FP64) | plans x2 | tile prefixes x2 | norms |
// conversion tables x4 | one slab per pair], as the forward batch; the single
// tier evaluates pairs with s > 0 in FP64 from FP64 copies of A and G.
template <typename T>
struct BVLayout {
  using Hi = typename Wide<T>::type;
  static constexpr bool kSplit = !std::is_same<T, Hi>::value;
  std::size_t items_lo = 0, items_hi = 0, plans_lo = 0, plans_hi = 0, prefix_lo = 0, prefix_hi = 0,
              prefix128 = 0, err = 0, norms = 0, conv = 0, total = 0;
  std::vector<std::size_t> slab;
  static std::size_t slab_bytes(int n) {
    if (!kSplit) return vslab_of<T>(n);
    const std::size_t nn = (std::size_t)n * n;
    return std::max(vslab_of<T>(n), vslab_of<Hi>(n) + 4 * align_up(nn * sizeof(Hi), 256));
  }
  void plan(int batch, const int *h_n) {
    Layout L(nullptr);
    items_lo = L.used;  L.take<BVItem<T, Hi>>(batch);
    items_hi = L.used;  L.take<BVItem<Hi, Hi>>(kSplit ? batch : 0);
    plans_lo = L.used;  L.take<BPlan>(batch);
    plans_hi = L.used;  L.take<BPlan>(kSplit ? batch : 0);
    prefix_lo = L.used; L.take<int>(batch + 1);
    prefix_hi = L.used; L.take<int>(kSplit ? batch + 1 : 0);
    prefix128 = L.used; L.take<int>(batch + 1);
    err = L.used;       L.take<int>(1);
    norms = L.used;     L.take<double>(batch);
    conv = L.used;      L.take<BConv>(kSplit ? 4 * (std::size_t)batch : 0);
    slab.resize(batch);
    std::size_t at = L.used;
    for (int i = 0; i < batch; ++i) {
      slab[i] = at;
      at += slab_bytes(h_n[i]);
    }
    total = at;
  }
};

template <typename T>
calamanStatus_t vjp_batched_api(calamanHandle_t blas, calamanStream_t stream, int batch, const int *h_n,
                                const T *const *h_A, const int *h_lda, const T *const *h_G,
                                const int *h_ldg, T *const *h_D, const int *h_ldd, T *const *h_E,
                                const int *h_lde, void *work, std::size_t lwork, int *d_info,
                                calamanExpmPlan_t *h_plans) {
  using R = typename elem<T>::real;
  using Hi = typename Wide<T>::type;
  using Lay = BVLayout<T>;
  if (batch < 0) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (batch == 0) return ok_status();
  if (h_n == nullptr || h_A == nullptr || h_lda == nullptr || h_G == nullptr || h_ldg == nullptr ||
      h_D == nullptr || h_ldd == nullptr || work == nullptr || d_info == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  for (int i = 0; i < batch; ++i) {
    const int n = h_n[i];
    const bool want_e = h_E != nullptr && h_E[i] != nullptr;
    if (n < 1 || h_lda[i] < n || h_ldg[i] < n || h_ldd[i] < n || h_A[i] == nullptr ||
        h_G[i] == nullptr || h_D[i] == nullptr || (want_e && (h_lde == nullptr || h_lde[i] < n)))
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    if (n > kBatchedMaxN) return blas_status(CALAMAN_STATUS_NOT_SUPPORTED);
  }
  Lay lay;
  lay.plan(batch, h_n);
  if (lwork < lay.total) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  PointerModeScope pm(blas);
  TimerScope ts(timer_of(blas));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int dev = 0;
  CLM_CUDA(cudaGetDevice(&dev));
  CLM_CUDA(upload_pade_table(dev));

  char *base = static_cast<char *>(work);
  auto *d_lo = reinterpret_cast<BVItem<T, Hi> *>(base + lay.items_lo);
  auto *d_hi = reinterpret_cast<BVItem<Hi, Hi> *>(base + lay.items_hi);
  auto *d_plo = reinterpret_cast<BPlan *>(base + lay.plans_lo);
  auto *d_phi = reinterpret_cast<BPlan *>(base + lay.plans_hi);
  auto *d_xlo = reinterpret_cast<int *>(base + lay.prefix_lo);
  auto *d_xhi = reinterpret_cast<int *>(base + lay.prefix_hi);
  auto *d_norms = reinterpret_cast<double *>(base + lay.norms);
  auto *d_conv = reinterpret_cast<BConv *>(base + lay.conv);

  std::vector<BVItem<T, Hi>> lo(batch);
  for (int i = 0; i < batch; ++i) {
    BVItem<T, Hi> &it = lo[i];
    carve_vitem<T>(it, base + lay.slab[i], h_n[i]);
    it.A = h_A[i];
    it.G = h_G[i];
    it.Dg = h_D[i];
    it.E = (h_E != nullptr) ? h_E[i] : nullptr;
    it.lda = h_lda[i];
    it.ldg = h_ldg[i];
    it.ldd = h_ldd[i];
    it.lde = it.E ? h_lde[i] : 0;
    it.id = i;
  }
  CLM_CUDA(cudaMemcpyAsync(d_lo, lo.data(), sizeof(BVItem<T, Hi>) * batch, cudaMemcpyHostToDevice, st));
  b_norm_kernel<BVItem<T, Hi>><<<batch, 256, 0, st>>>(d_lo, d_norms);
  CLM_CUDA(launched());
  std::vector<double> norms(batch);
  CLM_CUDA(cudaMemcpyAsync(norms.data(), d_norms, sizeof(double) * batch, cudaMemcpyDeviceToHost, st));
  CLM_CUDA(cudaStreamSynchronize(st));
  std::vector<calamanExpmPlan_t> plans(batch);
  for (int i = 0; i < batch; ++i) {
    if (!std::isfinite(norms[i])) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    plans[i] = plan_for<R>((R)norms[i]);
  }
  if (h_plans)
    for (int i = 0; i < batch; ++i) h_plans[i] = plans[i];

  std::vector<BVItem<T, Hi>> lo_items;
  std::vector<BVItem<Hi, Hi>> hi_items;
  std::vector<BPlan> lo_plans, hi_plans;
  std::vector<int> lo_prefix(1, 0), hi_prefix(1, 0), lo_n, hi_n;
  std::vector<BConv> cin, cout;
  int lo_max_n = 0, hi_max_n = 0, lo_max_s = 0, hi_max_s = 0;
  // matrices in ascending n: the LU runs one launch per size class
  std::vector<int> order(batch);
  for (int i = 0; i < batch; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return h_n[x] < h_n[y]; });
  for (int i : order) {
    const calamanExpmPlan_t &p = plans[i];
    const BPlan bp{p.m, p.s, pade_num_powers(p.m), 0};
    const int n = h_n[i];
    if (!Lay::kSplit || p.s == 0) {
      lo_items.push_back(lo[i]);
      lo_plans.push_back(bp);
      lo_prefix.push_back(lo_prefix.back() + tiles_of(n));
      lo_n.push_back(n);
      lo_max_n = std::max(lo_max_n, n);
      lo_max_s = std::max(lo_max_s, p.s);
    } else {
      BVItem<Hi, Hi> it{};
      carve_vitem<Hi>(it, base + lay.slab[i], n);
      const std::size_t nn = (std::size_t)n * n, step = align_up(nn * sizeof(Hi), 256);
      char *extra = base + lay.slab[i] + vslab_of<Hi>(n);
      Hi *a64 = reinterpret_cast<Hi *>(extra), *g64 = reinterpret_cast<Hi *>(extra + step);
      Hi *d64 = reinterpret_cast<Hi *>(extra + 2 * step), *e64 = reinterpret_cast<Hi *>(extra + 3 * step);
      it.A = a64;
      it.G = g64;
      it.Dg = d64;
      it.E = lo[i].E ? e64 : nullptr;
      it.lda = it.ldg = it.ldd = it.lde = n;
      it.id = i;
      hi_items.push_back(it);
      hi_plans.push_back(bp);
      hi_prefix.push_back(hi_prefix.back() + tiles_of(n));
      hi_n.push_back(n);
      hi_max_n = std::max(hi_max_n, n);
      hi_max_s = std::max(hi_max_s, p.s);
      cin.push_back(BConv{h_A[i], a64, n, h_lda[i], n, 0});
      cin.push_back(BConv{h_G[i], g64, n, h_ldg[i], n, 0});
      cout.push_back(BConv{d64, h_D[i], n, n, h_ldd[i], 0});
      if (lo[i].E) cout.push_back(BConv{e64, lo[i].E, n, n, h_lde[i], 0});
    }
  }
  const int nlo = (int)lo_items.size(), nhi = (int)hi_items.size();
  // a mixed batch runs its FP64 pairs on the handle's side stream, beside the
  // FP32 ones (every table is uploaded on st before the fork)
  cudaStream_t side = nullptr;
  CLM_CUDA(side_stream(blas, nlo > 0 && nhi > 0, side));
  cudaStream_t sh = side ? side : st;
  if (nhi > 0) {
    const int nin = (int)cin.size(), nout = (int)cout.size();
    CLM_CUDA(cudaMemcpyAsync(d_hi, hi_items.data(), sizeof(BVItem<Hi, Hi>) * nhi, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_phi, hi_plans.data(), sizeof(BPlan) * nhi, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_xhi, hi_prefix.data(), sizeof(int) * (nhi + 1), cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_conv, cin.data(), sizeof(BConv) * nin, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_conv + nin, cout.data(), sizeof(BConv) * nout, cudaMemcpyHostToDevice, st));
    CLM_CUDA(side_fork(blas, st, side));
    const unsigned chunks = (unsigned)((hi_max_n * hi_max_n + kEwChunk - 1) / kEwChunk);
    b_conv_kernel<T, Hi><<<dim3((unsigned)nin, chunks), 256, 0, sh>>>(d_conv);
    CLM_CUDA(launched());
    CLM_CUDA(run_vjp_phases<Hi>(sh, d_hi, d_phi, d_xhi, nhi, hi_prefix.back(), hi_max_n, hi_max_s, d_info,
                                hi_n, hi_plans, nullptr, 0, nullptr, 0, 0, lu_fork(blas, 1, batch)));
    b_conv_kernel<Hi, T><<<dim3((unsigned)nout, chunks), 256, 0, sh>>>(d_conv + nin);
    CLM_CUDA(launched());
  }
  if (nlo > 0) {
    CLM_CUDA(cudaMemcpyAsync(d_lo, lo_items.data(), sizeof(BVItem<T, Hi>) * nlo, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_plo, lo_plans.data(), sizeof(BPlan) * nlo, cudaMemcpyHostToDevice, st));
    CLM_CUDA(cudaMemcpyAsync(d_xlo, lo_prefix.data(), sizeof(int) * (nlo + 1), cudaMemcpyHostToDevice, st));
    // FP32 pairs from the schedule's threshold on take the tensor cores
    const bool tc = std::is_same<T, float>::value;
    const BatchedTuning tune = blas ? blas->tune : default_batched_tuning();
    int tc_first = 0;
    while (tc && tc_first < nlo && lo_n[tc_first] < tune.fp32_tc_min_n) ++tc_first;
    std::vector<int> tc_prefix(1, 0);
    for (int i = tc_first; i < nlo; ++i) tc_prefix.push_back(tc_prefix.back() + tiles128_of(lo_n[i]));
    auto *d_x128 = reinterpret_cast<int *>(base + lay.prefix128);
    auto *d_err = reinterpret_cast<int *>(base + lay.err);
    if (tc) {
      CLM_CUDA(cudaMemcpyAsync(d_x128, tc_prefix.data(), sizeof(int) * tc_prefix.size(), cudaMemcpyHostToDevice,
                               st));
      CLM_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    }
    CLM_CUDA(run_vjp_phases<T>(st, d_lo, d_plo, d_xlo, nlo, lo_prefix.back(), lo_max_n, lo_max_s, d_info,
                               lo_n, lo_plans, tc ? d_x128 : nullptr, tc_prefix.back(), d_err, tc_first,
                               lo_prefix[tc_first], lu_fork(blas, 0, batch)));
  }
  CLM_CUDA(side_join(blas, st, side));
  return ok_status();
}

template <typename T>
calamanStatus_t vjp_batched_bytes(int batch, const int *h_n, std::size_t *bytes) {
  if (batch < 0 || bytes == nullptr || (batch > 0 && h_n == nullptr))
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  for (int i = 0; i < batch; ++i) {
    if (h_n[i] < 1) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
    if (h_n[i] > kBatchedMaxN) return blas_status(CALAMAN_STATUS_NOT_SUPPORTED);
  }
  BVLayout<T> lay;
  lay.plan(batch, h_n);
  *bytes = batch > 0 ? lay.total : 0;
  return ok_status();
}

// Deterministic test matrices for the tuner: count n x n matrices, entries
// uniform in (-1, 1) from a hash of (matrix, index), scaled to a 1-norm of
// about 4 (single-precision plan m = 9, s = 0).
__global__ void tune_fill_kernel(float *A, int count, int n) {
  const std::size_t total = (std::size_t)count * n * n;
  for (std::size_t i = blockIdx.x * (std::size_t)blockDim.x + threadIdx.x; i < total;
       i += (std::size_t)gridDim.x * blockDim.x) {
    unsigned h = (unsigned)(i * 2654435761u) ^ (unsigned)(i >> 32) ^ 0x9e3779b9u;
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    h *= 0x846ca68bu;
    h ^= h >> 16;
    const float u = (float)(h >> 8) * (2.0f / 16777216.0f) - 1.0f;
    A[i] = u * (8.0f / (float)n);
  }
}

// The batched schedule, measured: for every size bucket n = 16, 32, ..., 256
// a batch of `count` n x n float32 matrices runs through the mixed tier with
// every admissible per-matrix LU CTA size (64 / 128 / 256 threads, >= n) and
// both FP32 product engines (tensor cores, SIMT); the fastest configuration of
// each bucket is kept, and the FP32 engine threshold is the smallest n from
// which the tensor cores won every larger bucket.
calamanStatus_t tune_batched(calamanHandle_t h, int count, void *d_work, std::size_t work_bytes, int *lu_out,
                             int *tc_min_out) {
  cudaStream_t st = h->stream;
  const std::size_t mat = align_up((std::size_t)count * kBatchedMaxN * kBatchedMaxN * sizeof(float), 256);
  char *w = static_cast<char *>(d_work);
  float *A = reinterpret_cast<float *>(w);
  float *E = reinterpret_cast<float *>(w + mat);
  int *info = reinterpret_cast<int *>(w + 2 * mat);
  char *ws = w + 2 * mat + align_up((std::size_t)2 * count * sizeof(int), 256);
  const std::size_t ws_bytes = work_bytes - (std::size_t)(ws - w);
  const BatchedTuning saved = h->tune;
  const int saved_graphs = h->graphs;
  h->graphs = 0;
  BatchedTuning best = default_batched_tuning();
  bool tc_best[17] = {};
  cudaEvent_t a = nullptr, b = nullptr;
  CLM_CUDA(cudaEventCreate(&a));
  CLM_CUDA(cudaEventCreate(&b));
  calamanStatus_t status = ok_status();
  for (int bucket = 1; bucket <= 16 && is_ok(status); ++bucket) {
    const int n = 16 * bucket;
    std::vector<int> ns(count, n), lds(count, n);
    std::vector<const float *> pa(count);
    std::vector<float *> pe(count);
    for (int i = 0; i < count; ++i) {
      pa[i] = A + (std::size_t)i * n * n;
      pe[i] = E + (std::size_t)i * n * n;
    }
    tune_fill_kernel<<<4 * 148, 256, 0, st>>>(A, count, n);
    if (launched() != cudaSuccess) {
      status = runtime_status(cudaGetLastError());
      break;
    }
    float best_ms = 1e30f;
    for (int nt : {64, 128, 256}) {
      if (nt < n) continue;
      for (int eng = 0; eng < 2 && is_ok(status); ++eng) {
        BatchedTuning t = saved;
        t.lu_threads[bucket] = nt;
        t.fp32_tc_min_n = eng ? 1 : kBatchedMaxN + 1;
        h->tune = t;
        float ms = 0.f;
        for (int rep = 0; rep < 3 && is_ok(status); ++rep) {  // one warm-up, two timed
          if (rep == 1) cudaEventRecord(a, st);
          status = batched_api<float>(h, st, count, ns.data(), pa.data(), lds.data(), pe.data(), lds.data(), ws,
                                      ws_bytes, info, nullptr);
        }
        if (!is_ok(status)) break;
        cudaEventRecord(b, st);
        cudaEventSynchronize(b);
        cudaEventElapsedTime(&ms, a, b);
        if (ms < best_ms) {
          best_ms = ms;
          best.lu_threads[bucket] = nt;
          tc_best[bucket] = eng == 1;
        }
      }
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  h->graphs = saved_graphs;
  if (!is_ok(status)) {
    h->tune = saved;
    return status;
  }
  int min_n = kBatchedMaxN + 1;
  for (int bucket = 16; bucket >= 1 && tc_best[bucket]; --bucket) min_n = 16 * bucket - 15;
  best.fp32_tc_min_n = min_n;
  h->tune = best;
  if (lu_out)
    for (int bb = 0; bb <= 16; ++bb) lu_out[bb] = best.lu_threads[bb];
  if (tc_min_out) *tc_min_out = best.fp32_tc_min_n;
  return ok_status();
}

}  // namespace
}  // namespace clm

using namespace clm;

extern "C" {

calamanStatus_t calaman_expm_batched_bufferSize_s(calamanSolverHandle_t, int batch, const int *h_n,
                                                  size_t *bytes) {
  return batched_bytes<float>(batch, h_n, bytes);
}
calamanStatus_t calaman_expm_batched_bufferSize_d(calamanSolverHandle_t, int batch, const int *h_n,
                                                  size_t *bytes) {
  return batched_bytes<double>(batch, h_n, bytes);
}
calamanStatus_t calaman_expm_batched_s(calamanBlasHandle_t blas, calamanSolverHandle_t,
                                       calamanStream_t stream, int batch, const int *h_n,
                                       const float *const *h_A, const int *h_lda, float *const *h_E,
                                       const int *h_lde, void *d_work, size_t lwork, int *d_info,
                                       calamanExpmPlan_t *h_plans) {
  return batched_api<float>(blas, stream, batch, h_n, h_A, h_lda, h_E, h_lde, d_work, lwork, d_info,
                            h_plans);
}
calamanStatus_t calamanSetBatchedGraphs(calamanHandle_t handle, int enable) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  handle->graphs = enable != 0;
  return ok_status();
}

calamanStatus_t calamanGetBatchedGraphs(calamanHandle_t handle, int *enabled, int *cached) {
  if (handle == nullptr || enabled == nullptr || cached == nullptr)
    return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *enabled = handle->graphs;
  *cached = (handle->graph[0].exec != nullptr) + (handle->graph[1].exec != nullptr);
  return ok_status();
}

calamanStatus_t calamanSetBatchedTuning(calamanHandle_t handle, const int *lu_threads, int fp32_tc_min_n) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  BatchedTuning t = default_batched_tuning();
  if (lu_threads != nullptr)
    for (int b = 1; b <= 16; ++b) {
      const int v = lu_threads[b];
      if (!((v == 64 || v == 128 || v == 256) && v >= 16 * b)) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
      t.lu_threads[b] = v;
    }
  if (fp32_tc_min_n < 1) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  t.fp32_tc_min_n = fp32_tc_min_n;
  handle->tune = t;
  return ok_status();
}

calamanStatus_t calamanGetBatchedTuning(calamanHandle_t handle, int *lu_threads, int *fp32_tc_min_n) {
  if (handle == nullptr || lu_threads == nullptr || fp32_tc_min_n == nullptr)
    return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  for (int b = 0; b <= 16; ++b) lu_threads[b] = handle->tune.lu_threads[b];
  *fp32_tc_min_n = handle->tune.fp32_tc_min_n;
  return ok_status();
}

size_t calamanTuneBatched_bufferSize(int count) {
  if (count < 1) return 0;
  std::vector<int> ns(count, kBatchedMaxN);
  std::size_t wb = 0;
  batched_bytes<float>(count, ns.data(), &wb);
  const std::size_t mat = align_up((std::size_t)count * kBatchedMaxN * kBatchedMaxN * sizeof(float), 256);
  return 2 * mat + align_up((std::size_t)2 * count * sizeof(int), 256) + wb;
}

calamanStatus_t calamanTuneBatched(calamanHandle_t handle, int count, void *d_work, size_t work_bytes,
                                   int *lu_threads, int *fp32_tc_min_n) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (count < 1 || d_work == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (work_bytes < calamanTuneBatched_bufferSize(count)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  return tune_batched(handle, count, d_work, work_bytes, lu_threads, fp32_tc_min_n);
}

calamanStatus_t calaman_expm_batched_d(calamanBlasHandle_t blas, calamanSolverHandle_t,
                                       calamanStream_t stream, int batch, const int *h_n,
                                       const double *const *h_A, const int *h_lda, double *const *h_E,
                                       const int *h_lde, void *d_work, size_t lwork, int *d_info,
                                       calamanExpmPlan_t *h_plans) {
  return batched_api<double>(blas, stream, batch, h_n, h_A, h_lda, h_E, h_lde, d_work, lwork, d_info,
                             h_plans);
}

#define CLM_VJPB_API(SUF, T)                                                                       \
  calamanStatus_t calaman_expm_vjp_batched_bufferSize_##SUF(calamanSolverHandle_t, int batch,        \
                                                            const int *h_n, size_t *bytes) {         \
    return vjp_batched_bytes<T>(batch, h_n, bytes);                                                  \
  }                                                                                                  \
  calamanStatus_t calaman_expm_vjp_batched_##SUF(                                                    \
      calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream, int batch,            \
      const int *h_n, const T *const *h_A, const int *h_lda, const T *const *h_G, const int *h_ldg,   \
      T *const *h_gradA, const int *h_ldga, T *const *h_expA, const int *h_lde, void *d_work,        \
      size_t lwork, int *d_info, calamanExpmPlan_t *h_plans) {                                       \
    return vjp_batched_api<T>(blas, stream, batch, h_n, h_A, h_lda, h_G, h_ldg, h_gradA, h_ldga,     \
                              h_expA, h_lde, d_work, lwork, d_info, h_plans);                        \
  }
CLM_VJPB_API(s, float)
CLM_VJPB_API(d, double)
#undef CLM_VJPB_API

}  // extern "C"
