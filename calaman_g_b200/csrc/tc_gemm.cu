// tc_gemm.cu -- FP32 GEMM as split-BF16 products on the 5th-generation tensor
// cores (tcgen05, TMEM accumulators, TMA-fed shared memory), for the single-
// precision tiers of the matrix-exponential path.
//
// C = alpha * A B + beta * C with A (M x K), B (K x N), C column-major FP32.
// Each operand element x is split into bf16 parts
//     h = bf16(x), m = bf16(x - h), l = bf16(x - h - m)
// and the product is the sum of the part products the precision level keeps,
// smallest first, all accumulated into one FP32 accumulator in TMEM:
//     x3: (m,h) (h,m) (h,h)                          ~16-bit operands
//     x6: (l,h) (h,l) (m,m) (m,h) (h,m) (h,h)         ~24-bit operands
// Complex64 products are one real product of twice the rows and twice the
// depth, [Cr; Ci] = [[Ar, -Ai]; [Ai, Ar]] [Br; Bi]: the split kernels read the
// interleaved operands in that block form and the epilogue writes rows < M to
// the real and rows >= M to the imaginary halves of C.
// The parts are written once per operand by split kernels into a K-major
// layout (rows of Kpad bf16, zero padded to the tile grid), so the GEMM's
// producer warp reads every operand tile with one TMA copy, 128-byte swizzled.
//
// Kernel structure (one CTA per 128 x 256 output tile, 10 warps):
//   warp 0      TMA producer: a 4-stage ring of (A 128x64, B 256x64) tiles
//   warp 1      TMEM allocator and MMA issuer (one elected thread issues
//               tcgen05.mma 128x256x16, commits each stage back to the ring)
//   warps 2..9  epilogue, two warps per TMEM lane quarter: tcgen05.ld 32 lanes
//               x 32 columns at a time, alpha/beta, coalesced column-major
//               stores
// Every mbarrier wait is bounded; a wait that runs out records an error code
// and the CTA unwinds (draining its own TMA copies, freeing its TMEM).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace clm {

namespace {

using namespace tc;

constexpr int TM = 128;       // UMMA M (TMEM lanes)
constexpr int TN = 256;       // UMMA N (TMEM columns)
constexpr int TK = 64;        // k-block: one 128-byte swizzle atom of bf16
constexpr int UK = 16;        // UMMA K for 16-bit inputs
constexpr int kThreads = 320;   // producer, MMA issuer, 8 epilogue warps
constexpr int kA = TM * TK * 2;  // bytes of one A stage
constexpr int kB = TN * TK * 2;  // bytes of one B stage

struct TcParams {
  int M, N, nkb;        // nkb: k-blocks per part product (Kpad / TK); M: rows of the real product
  int Mc;               // complex: rows of the caller's C (rows >= Mc are imaginary parts), else 0
  int Mpad, Npad;       // rows of one A part / one B part in the part buffers
  int nterms;
  int pa[9], pb[9];     // part index of A and of B for every term
  float alpha, beta;
  float *C;
  int ldc;
  int *err;
};

// Instruction descriptor: bf16 x bf16 -> f32, both K-major, M = TM, N = TN.
constexpr uint32_t kIdesc = idesc_bf16_f32(TM, TN);

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc) {
  mma_f16(tmem_d, a, b, kIdesc, acc);
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) { mma_commit(bar); }
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) { return smem_desc_sw128(addr); }

// Element (m, n) of the real product in the caller's C, as a float index.
__device__ __forceinline__ std::size_t c_index(const TcParams &p, int m, int n) {
  if (p.Mc == 0) return (std::size_t)n * p.ldc + m;
  const bool im = m >= p.Mc;
  return 2 * ((std::size_t)n * p.ldc + (im ? m - p.Mc : m)) + (im ? 1 : 0);
}

constexpr int kStages = 4;  // depth of the TMA ring
__global__ void __launch_bounds__(kThreads, 1)
    tc_split_gemm_kernel(const __grid_constant__ CUtensorMap map_a,
                         const __grid_constant__ CUtensorMap map_b, const TcParams prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment for the 128-byte swizzle atoms
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *sA = base;
  unsigned char *sB = base + kStages * kA;
  uint64_t *full = reinterpret_cast<uint64_t *>(sB + kStages * kB);
  uint64_t *empty = full + kStages;
  uint64_t *acc_full = empty + kStages;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
  int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;
  const int total = prm.nterms * prm.nkb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // TMEM: 256 columns x 128 lanes of f32
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     saddr(tmem_slot)),
                 "r"(TN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    asm volatile("tcgen05.fence::before_thread_sync;");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- producer ----
    int issued = 0;
    for (int it = 0; it < total; ++it) {
      const int s = it % kStages;
      const uint32_t ph = (uint32_t)((it / kStages) & 1);
      if (!mbar_wait(&empty[s], ph ^ 1u) || *(volatile int *)abort_flag) {
        record_error(prm.err, 1);
        *(volatile int *)abort_flag = 1;
        break;
      }
      const int t = it / prm.nkb, kb = it - t * prm.nkb;
      mbar_expect_tx(&full[s], kA + kB);
      tma_load_2d(sA + s * kA, &map_a, &full[s], kb * TK, prm.pa[t] * prm.Mpad + m0);
      tma_load_2d(sB + s * kB, &map_b, &full[s], kb * TK, prm.pb[t] * prm.Npad + n0);
      issued = it + 1;
    }
    // drain: the copies this thread issued must land before the CTA exits
    for (int it = issued - kStages > 0 ? issued - kStages : 0; it < issued; ++it)
      mbar_wait(&full[it % kStages], (uint32_t)((it / kStages) & 1));
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer ----
    bool ok = true;
    for (int it = 0; it < total; ++it) {
      const int s = it % kStages;
      const uint32_t ph = (uint32_t)((it / kStages) & 1);
      if (!mbar_wait(&full[s], ph) || *(volatile int *)abort_flag) {
        record_error(prm.err, 2);
        *(volatile int *)abort_flag = 1;
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a0 = saddr(sA + s * kA), b0 = saddr(sB + s * kB);
#pragma unroll
      for (int k = 0; k < TK / UK; ++k)  // +32 bytes per 16-element k step inside the atom
        umma(tmem, smem_desc(a0 + k * 32), smem_desc(b0 + k * 32), (it > 0 || k > 0) ? 1u : 0u);
      umma_commit(&empty[s]);
    }
    if (!ok) *(volatile int *)abort_flag = 1;
    // The commit tracks every MMA issued above, so it is made on the abort
    // path too; this thread then waits for it, so no MMA still reads shared
    // memory or writes TMEM when the CTA frees its TMEM and exits.
    umma_commit(acc_full);
    if (!mbar_wait(acc_full, 0)) record_error(prm.err, 4);
  } else if (warp >= 2) {
    // ---- epilogue: two warps per TMEM lane quarter, 128 columns each ----
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;
    // bounded wait for the accumulator; gives up early once the CTA aborted
    bool ok = false;
    for (long long i = 0; i < kSpinLimit; ++i) {
      if (mbar_try_wait(acc_full, 0)) {
        ok = true;
        break;
      }
      if ((i & 1023) == 1023 && *(volatile int *)abort_flag) break;
    }
    if (!ok && !*(volatile int *)abort_flag) record_error(prm.err, 3);
    if (ok && !*(volatile int *)abort_flag) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int m = m0 + q * 32 + lane;
      for (int c0 = half * (TN / 2); c0 < (half + 1) * (TN / 2); c0 += 32) {
        if (n0 + c0 >= prm.N) break;
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
        if (m < prm.M) {
          // the 32 old C values of this chunk are loaded before any store
          float old[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int n = n0 + c0 + j;
            old[j] = (prm.beta != 0.f && n < prm.N) ? prm.C[c_index(prm, m, n)] : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int n = n0 + c0 + j;
            if (n < prm.N) {
              const float x = prm.alpha * __uint_as_float(v[j]);
              prm.C[c_index(prm, m, n)] = (prm.beta == 0.f) ? x : fmaf(prm.beta, old[j], x);
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN));
  }
}

// ---- operand split kernels --------------------------------------------------
// Eight values split into bf16 parts, packed 16 bytes a part.
__device__ __forceinline__ void split8(const float (&x)[8], uint4 (&part)[3]) {
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    const float r0 = x[2 * i] - __low2float(h), r1 = x[2 * i + 1] - __high2float(h);
    const __nv_bfloat162 m = __floats2bfloat162_rn(r0, r1);
    const __nv_bfloat162 l = __floats2bfloat162_rn(r0 - __low2float(m), r1 - __high2float(m));
    w[0][i] = *reinterpret_cast<const uint32_t *>(&h);
    w[1][i] = *reinterpret_cast<const uint32_t *>(&m);
    w[2][i] = *reinterpret_cast<const uint32_t *>(&l);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) part[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// Element (m, k) of the real A operand: A itself, or for complex (Mc > 0,
// Kc = the complex depth) the block [[Ar, -Ai]; [Ai, Ar]].
template <typename T>
__device__ __forceinline__ float a_at(const T *A, int lda, int Mc, int Kc, int m, int k) {
  if constexpr (std::is_same<T, float2>::value) {
    const bool lo = m < Mc, left = k < Kc;
    const float2 z = A[(std::size_t)(left ? k : k - Kc) * lda + (lo ? m : m - Mc)];
    return lo ? (left ? z.x : -z.y) : (left ? z.y : z.x);
  } else {
    return A[(std::size_t)k * lda + m];
  }
}

// A (M x K real rows; column-major, lda) -> parts[p][row][k], rows of Kpad,
// Mpad rows per part (multiples of 64): 64 x 64 through a shared tile, each
// thread then writes 16-byte pieces of 8 k (2-byte stores had held this kernel
// at half of the memory rate: 4096 x 4096 54 us -> 25 us; split_b 58 -> 25 us).
template <typename T>
__global__ void __launch_bounds__(256)
    split_a_kernel(int M, int K, const T *__restrict__ A, int lda, int Mc, int Kc, int Mpad, int Kpad, int nparts,
                   __nv_bfloat16 *__restrict__ parts) {
  __shared__ float tile[64][65];
  const int mb = blockIdx.x * 64, kb = blockIdx.y * 64, t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < 16; ++q) {  // read: consecutive m along the lanes
    const int r = t & 63, kk = (t >> 6) + 4 * q, m = mb + r, k = kb + kk;
    tile[kk][r] = (m < M && k < K) ? a_at<T>(A, lda, Mc, Kc, m, k) : 0.f;
  }
  __syncthreads();
  const std::size_t part_stride = (std::size_t)Mpad * Kpad;
#pragma unroll
  for (int q = 0; q < 2; ++q) {  // write: eight lanes to the 128 bytes of a row
    const int kg = (t & 7) * 8, r = (t >> 3) + 32 * q;
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = tile[kg + j][r];
    uint4 v[3];
    split8(x, v);
    __nv_bfloat16 *at = parts + (std::size_t)(mb + r) * Kpad + kb + kg;
    *reinterpret_cast<uint4 *>(at) = v[0];
    *reinterpret_cast<uint4 *>(at + part_stride) = v[1];
    if (nparts > 2) *reinterpret_cast<uint4 *>(at + 2 * part_stride) = v[2];
  }
}

// B (K x N real; column-major, ldb; for complex [Br; Bi] with Kc the complex
// depth) -> parts[p][col][k]: already K-contiguous, 8 k a thread.
template <typename T>
__global__ void __launch_bounds__(256)
    split_b_kernel(int K, int N, const T *__restrict__ B, int ldb, int Kc, int Npad, int Kpad, int nparts,
                   __nv_bfloat16 *__restrict__ parts) {
  const std::size_t part_stride = (std::size_t)Npad * Kpad;
  const int pieces = Kpad >> 3;  // per column
  const long long total = (long long)Npad * pieces;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int n = (int)(i / pieces), k0 = (int)(i - (long long)n * pieces) * 8;
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + j;
      x[j] = 0.f;
      if (k < K && n < N) {
        if constexpr (std::is_same<T, float2>::value) {
          const float2 z = B[(std::size_t)n * ldb + (k < Kc ? k : k - Kc)];
          x[j] = k < Kc ? z.x : z.y;
        } else {
          x[j] = B[(std::size_t)n * ldb + k];
        }
      }
    }
    uint4 v[3];
    split8(x, v);
    __nv_bfloat16 *at = parts + (std::size_t)n * Kpad + k0;
    *reinterpret_cast<uint4 *>(at) = v[0];
    *reinterpret_cast<uint4 *>(at + part_stride) = v[1];
    if (nparts > 2) *reinterpret_cast<uint4 *>(at + 2 * part_stride) = v[2];
  }
}

// ---- products of few k-blocks: the split inside the GEMM ---------------------
// C = alpha A B + beta C for a depth of at most kRankK real columns (the LU's
// trailing updates and the updates of the triangular solves). Such a product is
// bound by its passes over C, so the operands are split where they are used and
// never written out as parts: one CTA per 128 x 128 tile of C, eight warps that
// read the FP32 operands, split them and store the part tiles K-major and
// 128-byte swizzled; one thread issues the part products (128 x 128 x 16), the
// eight warps load their old C values and drain the accumulator (old C fetched
// ahead of the products took 64 registers and spilled: 47 us against 42 at
// 4096 x 4096 x 64). 96 KB of part tiles, two CTAs per SM.
// The wait between the two k-blocks has one outcome for the CTA: where it runs
// out, the part tiles are left alone, no further product is issued, C is not
// written, and the CTA waits once more, bounded, for the products it did issue
// before it frees its TMEM.
// Complex64 runs as the real product of twice the rows and depth with both
// interleaved, row 2i = Re, 2i + 1 = Im (depth alike), so that B and C are the
// caller's arrays read as floats and only A takes the block form
// [[Ar, -Ai], [Ai, Ar]] per element.
// 4096 x 4096 x 64 float32: 42 us against 62 for two split kernels and the GEMM
// over the parts; 777 x 777 x 64: 10 against 33; complex64 777 expm 3393 -> 3123 us.
constexpr int RN = 128;               // columns of C per CTA
constexpr int kRankThreads = 256;
constexpr int kRankK = 128;           // two k-blocks at most
constexpr int kPart = TM * TK * 2;    // bytes of one 128 x 64 bf16 part tile

struct RankParams {
  int M, N, K, nkb, terms;  // the real product
  float alpha, beta;
  const float *A, *B;
  float *C;
  long long lda, ldb, ldc;  // in floats (complex: twice the caller's)
  int *err;
  long long spin;  // tries of every wait
  int skip;        // self-test: no product is issued, so that the waits run out
};

// One 16-byte piece (8 consecutive k of one row) of every part tile.
__device__ __forceinline__ void store_parts(unsigned char *tile, int nparts, int row, int piece, const float (&x)[8]) {
  uint4 v[3];
  split8(x, v);
  unsigned char *at = tile + row * 128 + ((piece ^ (row & 7)) << 4);
  *reinterpret_cast<uint4 *>(at) = v[0];
  *reinterpret_cast<uint4 *>(at + kPart) = v[1];
  if (nparts > 2) *reinterpret_cast<uint4 *>(at + 2 * kPart) = v[2];
}

template <bool CPLX>
__global__ void __launch_bounds__(kRankThreads, 2) tc_rank_kernel(const RankParams prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *sA = base, *sB = base + 3 * kPart;
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * RN;
  const int nparts = prm.terms == 3 ? 2 : 3;

  if (tid == 0) {
    mbar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, RN);

  // C: warp w owns rows 32 (w & 3) .. of columns 64 (w >> 2) ..
  const int row = m0 + (warp & 3) * 32 + lane, col0 = n0 + (warp >> 2) * 64;
  float *const Cp = prm.C + (std::size_t)col0 * prm.ldc + row;

  const bool vec = (prm.ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(prm.B) & 15) == 0;
  uint32_t tmem = 0;
  bool ok = true;
  int kb = 0;
  for (; kb < prm.nkb; ++kb) {
    if (kb > 0) {  // the part tiles are free once the products over them are done
      ok = __syncthreads_and(mbar_wait(&done, (uint32_t)(kb - 1) & 1u, prm.spin));
      if (!ok) break;
    }
    const int k0 = kb * TK;
    // A: lanes along the rows, eight k each
#pragma unroll
    for (int q = 0; q < TM * 8 / kRankThreads; ++q) {
      const int it = tid + q * kRankThreads;
      const int r = it & (TM - 1), piece = it >> 7, m = m0 + r;
      float x[8];
      if constexpr (CPLX) {
        // depth 2 kc, 2 kc + 1 of row 2 i: Re, -Im of A(i, kc); of row 2 i + 1: Im, Re
        const int i = m >> 1;
        const bool im = m & 1;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int kc = (k0 + piece * 8) / 2 + e;
          const bool in = m < prm.M && 2 * kc < prm.K;
          const float2 z = in ? *reinterpret_cast<const float2 *>(prm.A + (std::size_t)kc * prm.lda + 2 * i)
                              : make_float2(0.f, 0.f);
          x[2 * e] = im ? z.y : z.x;
          x[2 * e + 1] = im ? z.x : -z.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int k = k0 + piece * 8 + e;
          x[e] = (m < prm.M && k < prm.K) ? prm.A[(std::size_t)k * prm.lda + m] : 0.f;
        }
      }
      store_parts(sA, nparts, r, piece, x);
    }
    // B: already contiguous along k
#pragma unroll
    for (int q = 0; q < RN * 8 / kRankThreads; ++q) {
      const int it = tid + q * kRankThreads;
      const int piece = it & 7, r = it >> 3, n = n0 + r, k = k0 + piece * 8;
      const float *src = prm.B + (std::size_t)n * prm.ldb + k;
      float x[8];
      if (vec && n < prm.N && k + 8 <= prm.K) {
        const float4 u = *reinterpret_cast<const float4 *>(src), v = *reinterpret_cast<const float4 *>(src + 4);
        x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = (n < prm.N && k + e < prm.K) ? src[e] : 0.f;
      }
      store_parts(sB, nparts, r, piece, x);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read what these stores wrote
    fence_before();
    __syncthreads();
    fence_after();
    tmem = tmem_slot;
    if (tid == 0 && !prm.skip) {
      constexpr uint32_t idesc = idesc_bf16_f32(TM, RN);
      const uint32_t a0 = saddr(sA), b0 = saddr(sB);
      // smallest part products first: x6 (l,h) (h,l) (m,m) (m,h) (h,m) (h,h), x3 the last three
      const uint32_t pa = 0x001102u, pb = 0x010120u;  // one hex digit a term, the first term lowest
      for (int t = 6 - prm.terms; t < 6; ++t) {
        const uint32_t at = a0 + ((pa >> (4 * t)) & 15u) * kPart, bt = b0 + ((pb >> (4 * t)) & 15u) * kPart;
#pragma unroll
        for (int k = 0; k < TK / UK; ++k)
          mma_f16(tmem, smem_desc(at + k * 32), smem_desc(bt + k * 32), idesc,
                  (kb > 0 || t > 6 - prm.terms || k > 0) ? 1u : 0u);
      }
      mma_commit(&done);
    }
  }
  // every product issued: kb commits were made
  ok = mbar_wait(&done, (uint32_t)(kb - 1) & 1u, prm.spin) && ok;
  if (!ok) record_error(prm.err, 5);
  fence_after();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float *const c = Cp + (std::size_t)(h * 32) * prm.ldc;
    const int live = row < prm.M ? prm.N - col0 - h * 32 : 0;  // columns of this half inside C
    float old[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) old[j] = (prm.beta != 0.f && j < live) ? c[(std::size_t)j * prm.ldc] : 0.f;
    uint32_t v[32];
    tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 64 + h * 32), v);
    if (ok) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < live) c[(std::size_t)j * prm.ldc] = fmaf(prm.beta, old[j], prm.alpha * __uint_as_float(v[j]));
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    fence_after();
    tmem_dealloc(tmem, RN);
  }
}

// ---- host side ----------------------------------------------------------------
// A row-major bf16 matrix of `rows` x `cols` (cols contiguous), boxes of box_rows x 64.
bool make_map(CUtensorMap *map, void *ptr, long long rows, long long cols, int box_rows) {
  return make_rowmajor_map_sw128(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, rows, cols * 2, box_rows);
}

struct SplitLayout {
  int Mpad, Npad, Kpad;
  std::size_t a_bytes, b_bytes, total;
};
SplitLayout split_layout(int M, int N, int K, int nparts) {
  SplitLayout L;
  L.Mpad = (M + TM - 1) / TM * TM;
  L.Npad = (N + TN - 1) / TN * TN;
  L.Kpad = (K + TK - 1) / TK * TK;
  L.a_bytes = align_up((std::size_t)nparts * L.Mpad * L.Kpad * 2, 256);
  L.b_bytes = align_up((std::size_t)nparts * L.Npad * L.Kpad * 2, 256);
  L.total = 256 + L.a_bytes + L.b_bytes;  // [error word | A parts | B parts]
  return L;
}

}  // namespace

EncodeTiledFn tensor_map_encoder() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

bool make_rowmajor_map_sw128(CUtensorMap *map, CUtensorMapDataType type, int elem_bytes, void *ptr,
                             long long rows, long long row_bytes, int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr || row_bytes % 16 != 0 || row_bytes < 128) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / elem_bytes), (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, type, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

std::size_t tc_gemm_workspace_bytes(int M, int N, int K, int terms, bool cplx) {
  return split_layout(cplx ? 2 * M : M, N, cplx ? 2 * K : K, terms == 3 ? 2 : 3).total;
}

namespace {
template <typename T>
cudaError_t tc_gemm_run(cudaStream_t s, int Mc, int N, int Kc, double alpha, const T *A, int lda, const T *B,
                        int ldb, double beta, float *C, int ldc, void *ws, std::size_t ws_bytes, int terms,
                        long long spin = 0, int skip = 0) {
  constexpr bool cplx = std::is_same<T, float2>::value;
  if (Mc <= 0 || N <= 0) return cudaSuccess;
  const int M = cplx ? 2 * Mc : Mc, K = cplx ? 2 * Kc : Kc;  // the real product
  const int nparts = terms == 3 ? 2 : 3;
  const SplitLayout L = split_layout(M, N, K > 0 ? K : 1, nparts);
  if (ws == nullptr || ws_bytes < L.total) return cudaErrorInvalidValue;
  // shallower than the output, or added to it: the LU's and the solves' updates
  if (K <= kRankK && (beta != 0.0 || M > K || N > K)) {
    RankParams r = {};
    r.M = M, r.N = N, r.K = K, r.nkb = K > TK ? 2 : 1, r.terms = terms == 3 ? 3 : 6;
    r.alpha = (float)alpha, r.beta = (float)beta;
    r.A = reinterpret_cast<const float *>(A), r.B = reinterpret_cast<const float *>(B), r.C = C;
    const long long f = cplx ? 2 : 1;
    r.lda = f * lda, r.ldb = f * ldb, r.ldc = f * ldc;
    r.err = static_cast<int *>(ws);
    r.spin = spin > 0 ? spin : kSpinLimit;
    r.skip = skip;
    constexpr int smem = 6 * kPart + 1024;
    auto kern = tc_rank_kernel<cplx>;
    static OncePerDevice once;
    const cudaError_t e = opt_in_smem(once, kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((M + TM - 1) / TM, (N + RN - 1) / RN), kRankThreads, smem, s>>>(r);
    return launched();
  }
  char *w = static_cast<char *>(ws);
  int *err = reinterpret_cast<int *>(w);
  auto *pa = reinterpret_cast<__nv_bfloat16 *>(w + 256);
  auto *pb = reinterpret_cast<__nv_bfloat16 *>(w + 256 + L.a_bytes);

  cudaError_t e;
  split_a_kernel<T><<<dim3(L.Mpad / 64, L.Kpad / 64), 256, 0, s>>>(M, K, A, lda, Mc, Kc, L.Mpad, L.Kpad, nparts,
                                                                   pa);
  if ((e = launched()) != cudaSuccess) return e;
  const long long pieces = (long long)L.Npad * (L.Kpad / 8);
  split_b_kernel<T><<<(unsigned)std::min<long long>((pieces + 255) / 256, 1 << 20), 256, 0, s>>>(
      K, N, B, ldb, Kc, L.Npad, L.Kpad, nparts, pb);
  if ((e = launched()) != cudaSuccess) return e;

  CUtensorMap ma, mb;
  if (!make_map(&ma, pa, (long long)nparts * L.Mpad, L.Kpad, TM)) return cudaErrorNotSupported;
  if (!make_map(&mb, pb, (long long)nparts * L.Npad, L.Kpad, TN)) return cudaErrorNotSupported;

  TcParams p = {};
  p.M = M;
  p.Mc = cplx ? Mc : 0;
  p.N = N;
  p.nkb = L.Kpad / TK;
  p.Mpad = L.Mpad;
  p.Npad = L.Npad;
  if (terms == 3) {
    const int A3[3] = {1, 0, 0}, B3[3] = {0, 1, 0};
    p.nterms = 3;
    for (int t = 0; t < 3; ++t) p.pa[t] = A3[t], p.pb[t] = B3[t];
  } else {
    const int A6[6] = {2, 0, 1, 1, 0, 0}, B6[6] = {0, 2, 1, 0, 1, 0};
    p.nterms = 6;
    for (int t = 0; t < 6; ++t) p.pa[t] = A6[t], p.pb[t] = B6[t];
  }
  p.alpha = (float)alpha;
  p.beta = (float)beta;
  p.C = C;
  p.ldc = ldc;
  p.err = err;

  constexpr int smem = kStages * (kA + kB) + 1024 + 256;
  static OncePerDevice once;
  if ((e = opt_in_smem(once, tc_split_gemm_kernel, smem)) != cudaSuccess) return e;
  tc_split_gemm_kernel<<<dim3(L.Mpad / TM, L.Npad / TN), kThreads, smem, s>>>(ma, mb, p);
  return launched();
}
}  // namespace

cudaError_t tc_gemm_f32(cudaStream_t s, int M, int N, int K, double alpha, const float *A, int lda,
                        const float *B, int ldb, double beta, float *C, int ldc, void *ws,
                        std::size_t ws_bytes, int terms, long long spin, int skip) {
  return tc_gemm_run<float>(s, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, ws, ws_bytes, terms, spin, skip);
}

cudaError_t tc_gemm_c64(cudaStream_t s, int M, int N, int K, double alpha, const float2 *A, int lda,
                        const float2 *B, int ldb, double beta, float2 *C, int ldc, void *ws,
                        std::size_t ws_bytes, int terms) {
  return tc_gemm_run<float2>(s, M, N, K, alpha, A, lda, B, ldb, beta, reinterpret_cast<float *>(C), ldc, ws,
                             ws_bytes, terms);
}

}  // namespace clm
