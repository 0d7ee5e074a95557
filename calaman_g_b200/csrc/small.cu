// small.cu -- expm of one small matrix (n <= 64, complex n <= 48) in one
// kernel on one CTA: scaling, the Pade powers and combinations, the solve with
// partial pivoting and the squarings, all in shared memory.
//
// At these sizes the general path is about twenty launches of 2 to 30 us each
// that do no more than a few thousand operations per thread (float64 40 x 40:
// 115 us of kernels). One CTA does the same work with barriers in the place of
// launches, and is bound by their latency. The limit is the shared memory that
// six FP64 matrices take; beyond it the products belong on more than one SM.
// float64 40 x 40 from Python, the norm's readback included: 139 -> 81 us.
#include <algorithm>
#include <type_traits>

#include "expm_common.cuh"
#include "lu_panel.cuh"

namespace clm {
namespace {

constexpr int kSmallThreads = 256;

struct PadeTable {
  double b[14];
};

// R: ceil(n / 16). Matrices are NP x NP (NP = 16 R), column-major with columns
// PT = NP + 1 apart, zero beyond n, so no product needs bounds.
template <int R> struct SmallShape {
  static constexpr int NP = 16 * R, PT = NP + 1;
};

// acc[a][b] += row tx + 16 a of A times column ty + 16 b of B
template <typename U, int R>
__device__ __forceinline__ void small_mm(const U *A, const U *B, int n, int tx, int ty, U (&acc)[R][R]) {
  constexpr int PT = SmallShape<R>::PT;
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    U av[R], bv[R];
#pragma unroll
    for (int a = 0; a < R; ++a) av[a] = A[k * PT + tx + 16 * a];
#pragma unroll
    for (int b = 0; b < R; ++b) bv[b] = B[(ty + 16 * b) * PT + k];
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
      for (int b = 0; b < R; ++b) acc[a][b] = fmac(av[a], bv[b], acc[a][b]);
  }
}
template <typename U, int R>
__device__ __forceinline__ void small_clear(U (&acc)[R][R]) {
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) acc[a][b] = elem<U>::zero();
}

__device__ __forceinline__ double load_wide(float x) { return x; }
__device__ __forceinline__ double load_wide(double x) { return x; }
__device__ __forceinline__ double2 load_wide(float2 x) { return make_double2(x.x, x.y); }
__device__ __forceinline__ double2 load_wide(double2 x) { return x; }
template <typename T, typename U> __device__ __forceinline__ T store_as(U x) {
  if constexpr (std::is_same<T, float>::value) return (float)x;
  else if constexpr (std::is_same<T, float2>::value) return make_float2((float)x.x, (float)x.y);
  else return x;
}

// Solve q X = p with partial pivoting, q and p in shared memory, X column-major
// into out (columns PT apart). The 2 NP columns of [q | p] are eliminated
// together, so L is never kept: thread (i, g) holds row i's columns 4 t + g in
// registers, places turning by one every four steps so that the pivot column of
// step k is place 0 of group k & 3. Rows carry positions (ties go to the first
// position, as IxAMAX); a pivot row leaves for rows (U | Y), from which the
// back-substitution reads, thread (j, g) keeping rows 4 t + g of column j.
template <typename T, int R>
__device__ void small_solve(const T *q, const T *p, T *rows, T *out, int n, int *info) {
  constexpr int NP = SmallShape<R>::NP, PT = SmallShape<R>::PT;
  constexpr int P = 8 * R;                // places: 2 NP columns over four groups
  constexpr int RP = 2 * NP + 1;          // pitch of a stored row; column c at (c & 3) P + (c >> 2)
  constexpr int V = 16 / (int)sizeof(T);  // elements per 16-byte piece
  __shared__ __align__(16) T cur[2][4][P];
  __shared__ T col[2][64];
  __shared__ T rcp[2], rdiag[64];
  __shared__ int how_s[2];
  __shared__ unsigned key_s[2][2][2];
  __shared__ int pos_s[2][2];
  const int tid = threadIdx.x, i = tid & 63, g = tid >> 6, lane = tid & 31;
  T r[P];
#pragma unroll
  for (int t = 0; t < P; ++t) {
    const int c = 4 * t + g;
    r[t] = i < n ? (c < NP ? q[c * PT + i] : p[(c - NP) * PT + i]) : elem<T>::zero();
  }
  bool active = i < n;
  int pos = i, first_zero = -1;
  __syncthreads();  // rows may overlap nothing that is still being read
#pragma unroll 1
  for (int b = 0; 4 * b < n; ++b) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int k = 4 * b + s, par = s & 1;
      if (k < n) {
        if (g == s) {
          const PivotCand c = warp_best<T>(pivot_cand<T>(r[0], pos, active));
          if (lane == 0) {
            key_s[par][i >> 5][0] = c.hi;
            key_s[par][i >> 5][1] = c.lo;
            pos_s[par][i >> 5] = c.pos;
          }
          col[par][i] = r[0];
        }
        __syncthreads();
        const unsigned long long k0 = ((unsigned long long)key_s[par][0][0] << 32) | key_s[par][0][1];
        const unsigned long long k1 = ((unsigned long long)key_s[par][1][0] << 32) | key_s[par][1][1];
        const int p0 = pos_s[par][0], p1 = pos_s[par][1];
        const bool second = k1 > k0 || (k1 == k0 && p1 < p0);
        const unsigned long long key = second ? k1 : k0;
        const int win = second ? p1 : p0;
        if (active && pos == win) {
#pragma unroll
          for (int t = 0; t < P; t += V) {
            union {
              T e[V];
              uint4 u;
            } w;
#pragma unroll
            for (int e = 0; e < V; ++e) w.e[e] = r[t + e];
            *reinterpret_cast<uint4 *>(&cur[par][g][t]) = w.u;
          }
#pragma unroll
          for (int t = 0; t < P; ++t)
            if (t + b < P) rows[k * RP + g * P + t + b] = r[t];
          if (g == s) {
            const bool zero = key == 0ull || is_zero(r[0]);
            how_s[par] = zero ? kScaleNone : abs1(r[0]) >= safe_min<T>() ? kScaleReciprocal : kScaleDivide;
            rcp[par] = zero ? elem<T>::one() : divide(elem<T>::one(), r[0]);
          }
        }
        __syncthreads();
        const int how = how_s[par];
        if (how == kScaleNone && first_zero < 0) first_zero = k;
        if (active) {
          if (pos == win) {
            active = false;
          } else {
            if (pos == k) pos = win;
            const T x = col[par][i];
            const T l = how == kScaleReciprocal ? mul(x, rcp[par])
                        : how == kScaleDivide   ? divide(x, cur[par][s][0])
                                                : x;
#pragma unroll
            for (int t = 0; t < P; t += V) {
              union {
                T e[V];
                uint4 u;
              } w;
              w.u = *reinterpret_cast<const uint4 *>(&cur[par][g][t]);
#pragma unroll
              for (int e = 0; e < V; ++e)
                if (t + e > 0 || g > s) r[t + e] = sub(r[t + e], mul(l, w.e[e]));
            }
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t + 1 < P; ++t) r[t] = r[t + 1];
  }
  if (tid == 0) {
    info[0] = first_zero >= 0 ? first_zero + 1 : 0;
    info[1] = 0;
  }
  __syncthreads();
  auto at = [&](int row, int c) -> T { return rows[row * RP + (c & 3) * P + (c >> 2)]; };
  if (tid < n) rdiag[tid] = divide(elem<T>::one(), at(tid, tid));
  __syncthreads();

  constexpr int PB = NP / 4;
  const int j = tid >> 2, bg = tid & 3, B = (n + 3) / 4;
  T y[PB];
#pragma unroll
  for (int t = 0; t < PB; ++t) {
    const int row = 4 * (t - PB + B) + bg;
    y[t] = (row >= 0 && row < n && j < NP) ? at(row, NP + j) : elem<T>::zero();
  }
#pragma unroll 1
  for (int b = B - 1; b >= 0; --b) {
#pragma unroll
    for (int s = 3; s >= 0; --s) {
      const int k = 4 * b + s;
      if (k < n) {
        const T x = shfl(mul(y[PB - 1], rdiag[k]), (lane & ~3) | s);
        if (bg == s && j < NP) out[j * PT + k] = x;
        if (bg < s) y[PB - 1] = sub(y[PB - 1], mul(at(4 * b + bg, k), x));
#pragma unroll
        for (int t = 0; t + 1 < PB; ++t)
          if (t - PB + 1 + b >= 0) y[t] = sub(y[t], mul(at(4 * (t - PB + 1 + b) + bg, k), x));
      }
    }
#pragma unroll
    for (int t = PB - 1; t > 0; --t) y[t] = y[t - 1];
  }
  __syncthreads();
}

// TI: the caller's type. The evaluation is FP64 throughout, the single tiers
// included: nothing here is bound by the arithmetic, and their result is then
// rounded once.
template <typename TI, int R>
__global__ void __launch_bounds__(kSmallThreads, 1)
    expm_small_kernel(int n, const TI *__restrict__ A, int lda, TI *E, int lde, int m, int s, PadeTable tab,
                      int *__restrict__ info) {
  using T = typename Wide<TI>::type;
  using Re = double;
  constexpr int NP = SmallShape<R>::NP, PT = SmallShape<R>::PT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *const buf = reinterpret_cast<T *>(smem_raw);
  constexpr int kBuf = NP * PT;
  T *const X = buf, *const P2 = buf + kBuf, *const P4 = buf + 2 * kBuf, *const P6 = buf + 3 * kBuf,
          *const P8 = buf + 4 * kBuf, *const Wm = buf + 5 * kBuf;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const double f = ldexp(1.0, -s);
  for (int e = tid; e < NP * NP; e += kSmallThreads) {
    const int c = e / NP, r = e % NP;
    X[c * PT + r] = (r < n && c < n) ? scale(load_wide(A[(std::size_t)c * lda + r]), f) : elem<T>::zero();
  }
  __syncthreads();

  T acc[R][R];
  auto product = [&](const T *Ab, const T *Bb, T *C) {  // C is none of the operands
    small_clear<T, R>(acc);
    small_mm<T, R>(Ab, Bb, n, tx, ty, acc);
    if (C != nullptr) {
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) C[(ty + 16 * b) * PT + tx + 16 * a] = acc[a][b];
    }
    __syncthreads();
  };
  // b_i0 P2 + b_i1 P4 + ... (+ b_d I) at this thread's element (a, b); zero beyond n
  auto combine = [&](int a, int b, Re c2, Re c4, Re c6, Re c8, Re cd, bool with8) -> T {
    const int row = tx + 16 * a, c = ty + 16 * b, e = c * PT + row;
    T v = scale(P2[e], c2);
    v = rfma(c4, P4[e], v);
    v = rfma(c6, P6[e], v);
    if (with8) v = rfma(c8, P8[e], v);
    if (row == c && row < n) v = add_real(v, cd);
    return v;
  };
  auto fill = [&](T *C) {  // powers that the degree does without read as zero
    for (int e = tid; e < kBuf; e += kSmallThreads) C[e] = elem<T>::zero();
  };
  const double *b = tab.b;
  const int np = m == 13 ? 3 : (m - 1) / 2;
  if (np < 2) fill(P4);
  if (np < 3) fill(P6);
  if (np < 4 && m != 13) fill(P8);
  product(X, X, P2);
  if (np >= 2) product(P2, P2, P4);
  if (np >= 3) product(P4, P2, P6);
  if (np >= 4) product(P4, P4, P8);

  T v[R][R];
  if (m == 13) {
    auto pass = [&](Re t2, Re t4, Re t6, Re c2, Re c4, Re c6, Re cd) {  // v = combination + P6 (t2 P2 + t4 P4 + t6 P6)
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int c = 0; c < R; ++c)
          P8[(ty + 16 * c) * PT + tx + 16 * a] = combine(a, c, t2, t4, t6, (Re)0, (Re)0, false);
      __syncthreads();
      product(P6, P8, nullptr);
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int c = 0; c < R; ++c) v[a][c] = add(combine(a, c, c2, c4, c6, (Re)0, cd, false), acc[a][c]);
    };
    pass((Re)b[9], (Re)b[11], (Re)b[13], (Re)b[3], (Re)b[5], (Re)b[7], (Re)b[1]);
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
      for (int c = 0; c < R; ++c) Wm[(ty + 16 * c) * PT + tx + 16 * a] = v[a][c];
    pass((Re)b[8], (Re)b[10], (Re)b[12], (Re)b[2], (Re)b[4], (Re)b[6], (Re)b[0]);
  } else {
    // coefficients past the degree are zero in the table
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
      for (int c = 0; c < R; ++c) {
        v[a][c] = combine(a, c, (Re)b[2], (Re)b[4], (Re)b[6], (Re)b[8], (Re)b[0], true);
        Wm[(ty + 16 * c) * PT + tx + 16 * a] = combine(a, c, (Re)b[3], (Re)b[5], (Re)b[7], (Re)b[9], (Re)b[1], true);
      }
    __syncthreads();
  }
  product(X, Wm, nullptr);  // U; every read of the powers is behind its barrier
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int e = (ty + 16 * c) * PT + tx + 16 * a;
      P2[e] = sub(v[a][c], acc[a][c]);  // q
      P4[e] = add(v[a][c], acc[a][c]);  // p
    }
  __syncthreads();
  small_solve<T, R>(P2, P4, P6, X, n, info);  // rows (U | Y) over P6 and P8

  if (s == 0) {
    for (int e = tid; e < n * NP; e += kSmallThreads) {
      const int c = e / NP, r = e % NP;
      if (r < n) E[(std::size_t)c * lde + r] = store_as<TI>(X[c * PT + r]);
    }
    return;
  }
  // squarings in place, through registers
#pragma unroll 1
  for (int k = 0; k < s; ++k) {
    product(X, X, nullptr);
    if (k + 1 < s) {
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int c = 0; c < R; ++c) X[(ty + 16 * c) * PT + tx + 16 * a] = acc[a][c];
      __syncthreads();
    }
  }
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int row = tx + 16 * a, cc = ty + 16 * c;
      if (row < n && cc < n) E[(std::size_t)cc * lde + row] = store_as<TI>(acc[a][c]);
    }
}

template <typename T, int R>
cudaError_t launch_small(cudaStream_t st, int n, const T *A, int lda, T *E, int lde, int m, int s, const PadeTable &tab,
                         int *info) {
  constexpr int smem = 6 * SmallShape<R>::NP * SmallShape<R>::PT * (int)sizeof(typename Wide<T>::type);
  auto kern = expm_small_kernel<T, R>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  kern<<<1, kSmallThreads, smem, st>>>(n, A, lda, E, lde, m, s, tab, info);
  return launched();
}

}  // namespace

template <typename T>
int expm_small_max_n() {
  return elem<T>::complex ? 48 : 64;
}

template <typename T>
cudaError_t expm_small(cudaStream_t st, int n, const T *A, int lda, T *E, int lde, int m, int s, int *info) {
  PadeTable tab = {};
  std::copy(pade_coeffs(m), pade_coeffs(m) + m + 1, tab.b);
  if (n <= 16) return launch_small<T, 1>(st, n, A, lda, E, lde, m, s, tab, info);
  if (n <= 32) return launch_small<T, 2>(st, n, A, lda, E, lde, m, s, tab, info);
  if (n <= 48) return launch_small<T, 3>(st, n, A, lda, E, lde, m, s, tab, info);
  if constexpr (!elem<T>::complex)
    if (n <= 64) return launch_small<T, 4>(st, n, A, lda, E, lde, m, s, tab, info);
  return cudaErrorInvalidValue;
}

#define CLM_INST_SMALL(T)                                                                                   \
  template int expm_small_max_n<T>();                                                                       \
  template cudaError_t expm_small<T>(cudaStream_t, int, const T *, int, T *, int, int, int, int *);
CLM_INST_SMALL(float)
CLM_INST_SMALL(double)
CLM_INST_SMALL(float2)
CLM_INST_SMALL(double2)
#undef CLM_INST_SMALL

}  // namespace clm
