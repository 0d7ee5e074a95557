// driver.cu -- host drivers of the matrix-exponential path and the C ABI.
//
// The drivers follow calaman_G's control flow step for step (file:line
// citations per function) but every kernel they enqueue is this library's own:
// the norm, Pade combinations and split from elementwise.cu, the tensor-core
// GEMMs from gemm.cu and the cluster LU from lu.cu.
#include <atomic>
#include <cstdio>
#include <cstring>
#include <utility>

#include "expm_common.cuh"
#include "graph_replay.cuh"

namespace clm {

unsigned long long g_launch_count();

namespace {

// ---- workspaces --------------------------------------------------------
// pade(): [P0 .. P_{np-1} | X (m = 13) | V | W | LU scratch | (FP32: tensor-core
// operand parts)], all 256-aligned. P0 doubles as U = A W and then as the
// numerator p = V + U; V becomes the denominator q = V - U and is factored in
// place (src/expm/detail.cppm:47-98).
template <typename T>
struct PadeWs {
  T *P[4] = {nullptr, nullptr, nullptr, nullptr};
  T *X = nullptr, *V = nullptr, *W = nullptr;
  void *lu = nullptr;
  void *tc = nullptr;
  std::size_t tc_bytes = 0;
  void *oz = nullptr;  // digit planes of the emulated FP64 products (oz_bytes > 0)
  std::size_t oz_bytes = 0;
  std::size_t carve(void *base, int n, int m, std::size_t ozb) {
    Layout L(base);
    const std::size_t nn = (std::size_t)n * n;
    const int np = pade_num_powers(m);
    for (int k = 0; k < np; ++k) P[k] = L.take<T>(nn);
    if (m == 13) X = L.take<T>(nn);
    V = L.take<T>(nn);
    W = L.take<T>(nn);
    lu = L.take<char>(lu_scratch_bytes(n));
    tc_bytes = tc_scratch_bytes<T>(n);
    if (tc_bytes) tc = L.take<char>(tc_bytes);
    oz_bytes = ozb;
    if (oz_bytes) oz = L.take<char>(oz_bytes);
    return L.used;
  }
};


// expm(): [As (also the squaring scratch) | colsum | norm | (single tiers: two
// FP64 n x n squaring buffers) | pade region]
template <typename T>
struct ExpmWs {
  using W = typename Wide<T>::type;
  T *As = nullptr;
  double *colsum = nullptr;
  double *norm = nullptr;
  W *wide = nullptr;
  void *pade = nullptr;
  std::size_t carve(void *base, int n) {
    Layout L(base);
    As = L.take<T>((std::size_t)n * n);
    colsum = L.take<double>(n);
    norm = L.take<double>(1);
    if (elem<T>::single) wide = L.take<W>(2 * (std::size_t)n * n);
    pade = L.cursor();
    return L.used;
  }
};

template <typename T>
std::size_t pade_bytes(calamanHandle_t h, int n, int m) {
  PadeWs<T> w;
  return w.carve(nullptr, n, m, oz_scratch_bytes<T>(h, n));
}

template <typename T>
std::size_t expm_bytes(calamanHandle_t h, int n) {
  ExpmWs<T> e;
  std::size_t worst = 0;
  for (int m : {3, 5, 7, 9, 13}) worst = std::max(worst, pade_bytes<T>(h, n, m));
  return e.carve(nullptr, n) + worst;
}

// ---- pade<T>, src/expm/pade.cppm:77-191 -------------------------------------
template <typename T>
calamanStatus_t pade_run(cudaStream_t st, int m, int n, const T *A, int lda, T *R, int ldr,
                         void *work, int *d_info, calamanHandle_t h) {
  const double *b = pade_coeffs(m);
  PadeWs<T> ws;
  ws.carve(work, n, m, oz_scratch_bytes<T>(h, n));
  GemmScratch gs = lend_scratch<T>(h, n, ws.tc, ws.tc_bytes, ws.oz, ws.oz_bytes);
  GemmScratchScope gss((ws.tc || ws.oz) ? &gs : nullptr);
  const int np = pade_num_powers(m);
  auto mm = [&](const T *X, int ldx, const T *Y, int ldy, double beta, T *Z) {
    return gemm_nn<T>(st, n, n, n, 1.0, X, ldx, Y, ldy, beta, Z, n);
  };
  CLM_CUDA(mm(A, lda, A, lda, 0.0, ws.P[0]));                      // A2
  if (np >= 2) CLM_CUDA(mm(ws.P[0], n, ws.P[0], n, 0.0, ws.P[1]));  // A4
  if (np >= 3) CLM_CUDA(mm(ws.P[1], n, ws.P[0], n, 0.0, ws.P[2]));  // A6
  if (np >= 4) CLM_CUDA(mm(ws.P[1], n, ws.P[1], n, 0.0, ws.P[3]));  // A8

  double cv[5] = {0, 0, 0, 0, 0}, cw[5] = {0, 0, 0, 0, 0};
  if (m != 13) {
    for (int i = 0; i <= np; ++i) {
      cv[i] = b[2 * i];
      cw[i] = b[2 * i + 1];
    }
    CLM_CUDA(launch_pade_even_odd<T>(st, n, np, ws.P[0], ws.P[1], ws.P[2], ws.P[3], cv, cw, ws.V, ws.W));
  } else {
    // odd parity: X = b9 A2 + b11 A4 + b13 A6, W = b1 I + b3 A2 + b5 A4 + b7 A6; W += A6 X
    const double cvo[5] = {0.0, b[9], b[11], b[13], 0.0};
    const double cwo[5] = {b[1], b[3], b[5], b[7], 0.0};
    CLM_CUDA(launch_pade_even_odd<T>(st, n, 3, ws.P[0], ws.P[1], ws.P[2], nullptr, cvo, cwo, ws.X, ws.W));
    CLM_CUDA(mm(ws.P[2], n, ws.X, n, 1.0, ws.W));
    // even parity: X = b8 A2 + b10 A4 + b12 A6, V = b0 I + b2 A2 + b4 A4 + b6 A6; V += A6 X
    const double cve[5] = {0.0, b[8], b[10], b[12], 0.0};
    const double cwe[5] = {b[0], b[2], b[4], b[6], 0.0};
    CLM_CUDA(launch_pade_even_odd<T>(st, n, 3, ws.P[0], ws.P[1], ws.P[2], nullptr, cve, cwe, ws.X, ws.V));
    CLM_CUDA(mm(ws.P[2], n, ws.X, n, 1.0, ws.V));
  }
  T *U = ws.P[0];
  CLM_CUDA(mm(A, lda, ws.W, n, 0.0, U));  // U = A W
  // p = V + U over U (the same thread reads then writes each element), q = V - U over V
  CLM_CUDA(launch_pade_split<T>(st, n, U, ws.V, U, n, ws.V));
  CLM_CUDA(getrf_solve<T>(st, n, ws.V, n, ws.lu, n, U, n, R, ldr, false, d_info));
  return ok_status();
}

template <typename T>
calamanStatus_t pade_api(calamanHandle_t blas, calamanStream_t stream, int m, int n, const T *A,
                         int lda, T *R, int ldr, void *work, std::size_t lwork, int *d_info) {
  if (pade_coeffs(m) == nullptr || n < 1 || n > kMaxDim || lda < n || ldr < n || work == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (lwork < pade_bytes<T>(blas, n, m)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  if (A == nullptr || R == nullptr || d_info == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  PointerModeScope pm(blas);
  TimerScope ts(timer_of(blas));
  return pade_run<T>(static_cast<cudaStream_t>(stream), m, n, A, lda, R, ldr, work, d_info, blas);
}

// ---- expm<T>, src/expm/expm.cppm:87-174 -------------------------------------
template <typename T>
calamanStatus_t expm_api(calamanHandle_t blas, calamanStream_t stream, int n, const T *A, int lda,
                         T *E, int lde, void *work, std::size_t lwork, int *d_info,
                         calamanExpmPlan_t *plan_out) {
  using R = typename elem<T>::real;
  if (n < 1 || n > kMaxDim || lda < n || lde < n || work == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (lwork < expm_bytes<T>(blas, n)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  if (A == nullptr || E == nullptr || d_info == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  PointerModeScope pm(blas);
  TimerScope ts(timer_of(blas));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ExpmWs<T> ws;
  ws.carve(work, n);

  // the norm the whole plan hangs off: FP64 sums on the device, one readback
  CLM_CUDA(launch_norm1<T>(st, n, A, lda, nullptr, ws.norm));
  double norm = 0.0;
  double *host = (blas && blas->h_pinned) ? blas->h_pinned : &norm;
  CLM_CUDA(cudaMemcpyAsync(host, ws.norm, sizeof(double), cudaMemcpyDeviceToHost, st));
  CLM_CUDA(cudaStreamSynchronize(st));
  norm = *host;
  if (!std::isfinite(norm)) return blas_status(CALAMAN_STATUS_INVALID_VALUE);

  const calamanExpmPlan_t chosen = plan_for<R>((R)norm);
  if (plan_out) *plan_out = chosen;

  // Small matrices: everything after the norm in one kernel, faster than the
  // general path's launches even as a graph (see small.cu). It has no GEMM launch
  // to time, and is the same with kernel timing on.
  if (n <= expm_small_max_n<T>()) {
    CLM_CUDA(expm_small<T>(st, n, A, lda, E, lde, chosen.m, chosen.s, d_info));
    return ok_status();
  }

  // everything after the plan: launches only, no host synchronisation
  auto post = [&]() -> calamanStatus_t {
    const T *src = A;
    int ld_src = lda;
    if (chosen.s > 0) {
      CLM_CUDA(launch_scale_copy<T>(st, n, std::ldexp(1.0, -chosen.s), A, lda, ws.As, n));
      src = ws.As;
      ld_src = n;
    }
    CLM_TRY(pade_run<T>(st, chosen.m, n, src, ld_src, E, lde, ws.pade, d_info, blas));

    // the squarings borrow the (now free) Pade region's digit planes
    PadeWs<T> pw;
    pw.carve(ws.pade, n, chosen.m, oz_scratch_bytes<T>(blas, n));
    GemmScratch gs = lend_scratch<T>(blas, n, nullptr, 0, pw.oz, pw.oz_bytes);
    GemmScratchScope gss(pw.oz ? &gs : nullptr);

    if (elem<T>::single && chosen.s > 0) {
      // single tiers: the squarings, where errors grow, run in FP64 tensor cores
      using W = typename Wide<T>::type;
      W *cw = ws.wide, *ow = ws.wide + (std::size_t)n * n;
      CLM_CUDA((launch_convert<T, W>(st, n, E, lde, cw, n)));
      for (int k = 0; k < chosen.s; ++k) {
        CLM_CUDA(gemm_nn<W>(st, n, n, n, 1.0, cw, n, cw, n, 0.0, ow, n));
        std::swap(cw, ow);
      }
      CLM_CUDA((launch_convert<W, T>(st, n, cw, n, E, lde)));
      return ok_status();
    }

    // square s times, ping-ponging between the output and the scratch
    T *cur = E, *other = ws.As;
    int ld_cur = lde, ld_other = n;
    for (int k = 0; k < chosen.s; ++k) {
      CLM_CUDA(gemm_nn<T>(st, n, n, n, 1.0, cur, ld_cur, cur, ld_cur, 0.0, other, ld_other));
      std::swap(cur, other);
      std::swap(ld_cur, ld_other);
    }
    if (cur != E) CLM_CUDA(launch_scale_copy<T>(st, n, 1.0, cur, ld_cur, E, lde));
    return ok_status();
  };
  // replayed as a CUDA graph while the configuration repeats
  CallKey key;
  key.mix((unsigned long long)n | ((unsigned long long)chosen.m << 32) | ((unsigned long long)chosen.s << 48));
  key.mix(A);
  key.mix((unsigned long long)lda | ((unsigned long long)lde << 32));
  key.mix(E);
  key.mix(work);
  key.mix((unsigned long long)lwork);
  key.mix(d_info);
  key.mix(st);
  if (blas == nullptr) return post();
  key.mix((unsigned long long)blas->split_terms | ((unsigned long long)(blas->fp64_digits + 16) << 32));
  key.mix(blas->work);
  key.mix((unsigned long long)blas->work_bytes);
  return run_or_replay(&blas->expm_graphs, blas->single[type_slot<T>()], st, key.h, post);
}

template <typename T, typename R>
R norm1_api(calamanStream_t stream, int n, const T *A, int lda, R *d_colsum) {
  if (n < 1 || lda < n || A == nullptr || d_colsum == nullptr) return (R)NAN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (launch_colsums_then_max<T, R>(st, n, A, lda, d_colsum) != cudaSuccess) return (R)NAN;
  R host = (R)NAN;
  if (cudaMemcpyAsync(&host, d_colsum, sizeof(R), cudaMemcpyDeviceToHost, st) != cudaSuccess) return (R)NAN;
  if (cudaStreamSynchronize(st) != cudaSuccess) return (R)NAN;
  return host;
}

// The horner / paterson_stockmeyer workspaces are sized exactly as the
// reference's (its tests pin them), so their FP32 products take the tensor
// cores only when the caller has attached a workspace to the handle
// (calamanSetWorkspace, as cublasSetWorkspace does): the split-BF16 operand
// parts live there. Without one they run on the SIMT kernel.
template <typename T>
GemmScratch handle_scratch(calamanHandle_t h) {
  GemmScratch gs;
  if (std::is_same<T, float>::value && h && h->work) {
    gs.ptr = h->work;
    gs.bytes = h->work_bytes;
    gs.terms = h->split_terms;
  }
  return gs;
}

// ---- horner<T>, src/horner/interface.cppm:104-194 ---------------------------
template <typename T>
std::size_t horner_bytes(int n) {
  const std::size_t order = (std::size_t)(n < 1 ? 1 : n);
  return align_up(order * order * sizeof(T), 256);
}

template <typename T>
calamanStatus_t horner_api(calamanHandle_t h, int n, const T *c, int degree, const T *A, int lda,
                           T *P, int ldp, void *work, std::size_t wbytes) {
  const calamanStatus_t bad = blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (!(n >= 1 && degree >= 0 && lda >= n && ldp >= n)) return bad;
  if (c == nullptr || A == nullptr || P == nullptr) return bad;
  if (!(degree == 0 || (work != nullptr && wbytes >= horner_bytes<T>(n)))) return bad;
  if (h == nullptr) return bad;
  TimerScope ts(timer_of(h));
  cudaStream_t st = h->stream;
  GemmScratch gs = handle_scratch<T>(h);
  GemmScratchScope gss(gs.ptr ? &gs : nullptr);
  T *buf[2] = {P, static_cast<T *>(work)};
  const int ld[2] = {ldp, n};
  int cur = (degree % 2 == 0) ? 0 : 1;
  CLM_CUDA(launch_set_scaled_identity<T>(st, buf[cur], n, ld[cur], c + degree));
  for (int k = degree - 1; k >= 0; --k) {
    const int next = 1 - cur;
    CLM_CUDA(gemm_nn<T>(st, n, n, n, 1.0, buf[cur], ld[cur], A, lda, 0.0, buf[next], ld[next]));
    cur = next;
    CLM_CUDA(launch_add_scaled_identity<T>(st, buf[cur], n, ld[cur], c + k));
  }
  return ok_status();
}

// ---- paterson_stockmeyer<T>, src/paterson_stockmeyer/interface.cppm:117-422 --
int ps_cost(int degree, int s) {
  if (s < 1 || degree < 1) return 0;
  const int r = degree / s;
  const int max_power = (r >= 1) ? s : degree;
  const int num_powers = (max_power >= 2) ? (max_power - 1) : 0;
  return num_powers + r;
}
int ps_block_size(int degree) {
  if (degree < 1) return 1;
  int best_s = 1, best = ps_cost(degree, 1);
  for (int s = 2; s <= degree + 1; ++s) {
    const int cst = ps_cost(degree, s);
    if (cst < best) {
      best = cst;
      best_s = s;
    }
  }
  return best_s;
}
calamanPatersonStockmeyerPlan_t ps_plan(int degree, int s_requested) {
  calamanPatersonStockmeyerPlan_t p{1, 0, 0, 0, 0};
  if (degree < 0) return p;
  int s = (s_requested > 0) ? s_requested : ps_block_size(degree);
  if (s > degree + 1) s = degree + 1;
  if (s < 1) s = 1;
  p.s = s;
  p.r = degree / s;
  const int max_power = (p.r >= 1) ? s : degree;
  p.num_powers = (max_power >= 2) ? (max_power - 1) : 0;
  p.num_blocks = p.num_powers + ((p.r >= 1) ? 1 : 0);
  p.num_gemms = p.num_powers + p.r;
  return p;
}
template <typename T>
std::size_t ps_stride(int n) {
  const std::size_t order = (std::size_t)(n < 1 ? 1 : n);
  return align_up(order * order * sizeof(T), 256) / sizeof(T);
}
template <typename T>
std::size_t ps_bytes(int n, int degree, int s_requested) {
  const int order = n < 1 ? 1 : n;
  const calamanPatersonStockmeyerPlan_t plan = ps_plan(degree, s_requested);
  Layout L(nullptr);
  if (plan.num_powers > 0) L.take<T>((std::size_t)plan.num_powers * ps_stride<T>(order));
  if (plan.r >= 1) L.take<T>((std::size_t)order * order);
  return L.used;
}

template <typename T>
calamanStatus_t ps_api(calamanHandle_t h, int n, const T *c, int degree, const T *A, int lda, T *P,
                       int ldp, void *work, std::size_t wbytes, int s_requested) {
  const calamanStatus_t bad = blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (n < 1 || degree < 0 || lda < n || ldp < n || s_requested < 0) return bad;
  if (c == nullptr || A == nullptr || P == nullptr) return bad;
  const calamanPatersonStockmeyerPlan_t plan = ps_plan(degree, s_requested);
  if (plan.num_blocks > 0 && (work == nullptr || wbytes < ps_bytes<T>(n, degree, s_requested)))
    return bad;
  if (h == nullptr) return bad;
  TimerScope ts(timer_of(h));
  cudaStream_t st = h->stream;
  GemmScratch gs = handle_scratch<T>(h);
  GemmScratchScope gss(gs.ptr ? &gs : nullptr);
  const std::size_t stride = ps_stride<T>(n);
  Layout L(work);
  T *powers = plan.num_powers > 0 ? L.take<T>((std::size_t)plan.num_powers * stride) : nullptr;
  T *scratch = plan.r >= 1 ? L.take<T>((std::size_t)n * n) : nullptr;
  // power bank: A^k = A^(k-1) A
  for (int k = 2; k <= plan.num_powers + 1; ++k) {
    const T *left = (k == 2) ? A : powers + (std::size_t)(k - 3) * stride;
    const int ldl = (k == 2) ? lda : n;
    CLM_CUDA(gemm_nn<T>(st, n, n, n, 1.0, left, ldl, A, lda, 0.0, powers + (std::size_t)(k - 2) * stride, n));
  }
  const bool have_x = plan.r >= 1;
  const T *X = !have_x ? nullptr : (plan.s >= 2 ? powers + (std::size_t)(plan.s - 2) * stride : A);
  const int ldx = (plan.s >= 2) ? n : lda;
  T *buf[2] = {P, scratch};
  const int ld[2] = {ldp, n};
  int cur = (plan.r % 2 == 0) ? 0 : 1;
  auto terms = [&](int j) {
    const int remaining = degree - j * plan.s + 1;
    return remaining < plan.s ? remaining : plan.s;
  };
  CLM_CUDA(launch_ps_build_block<T>(st, buf[cur], ld[cur], n, A, lda, powers, stride,
                                    c + (std::size_t)plan.r * plan.s, terms(plan.r)));
  for (int j = plan.r - 1; j >= 0; --j) {
    const int next = 1 - cur;
    CLM_CUDA(launch_ps_build_block<T>(st, buf[next], ld[next], n, A, lda, powers, stride,
                                      c + (std::size_t)j * plan.s, terms(j)));
    CLM_CUDA(gemm_nn<T>(st, n, n, n, 1.0, buf[cur], ld[cur], X, ldx, 1.0, buf[next], ld[next]));
    cur = next;
  }
  return ok_status();
}

}  // namespace

// The expm driver and its workspace size for callers in other translation
// units (the balanced composition in balance.cu).
template <typename T>
calamanStatus_t expm_entry(calamanHandle_t blas, calamanStream_t stream, int n, const T *A, int lda, T *E,
                           int lde, void *work, std::size_t lwork, int *d_info, calamanExpmPlan_t *plan) {
  return expm_api<T>(blas, stream, n, A, lda, E, lde, work, lwork, d_info, plan);
}
template <typename T>
std::size_t expm_workspace_bytes(calamanHandle_t h, int n) {
  return expm_bytes<T>(h, n);
}
#define CLM_INST_ENTRY(T)                                                                              \
  template calamanStatus_t expm_entry<T>(calamanHandle_t, calamanStream_t, int, const T *, int, T *, int, \
                                         void *, std::size_t, int *, calamanExpmPlan_t *);              \
  template std::size_t expm_workspace_bytes<T>(calamanHandle_t, int);
CLM_INST_ENTRY(float)
CLM_INST_ENTRY(double)
CLM_INST_ENTRY(float2)
CLM_INST_ENTRY(double2)
#undef CLM_INST_ENTRY

int sm_count() {
  int dev = 0, cnt = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&cnt, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return cnt;
}

namespace {
std::atomic<unsigned long long> g_launches{0};
}
void note_launch(unsigned n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
unsigned long long g_launch_count() { return g_launches.load(std::memory_order_relaxed); }

thread_local KernelTimer *tl_timer = nullptr;
thread_local GemmScratch *tl_gemm_scratch = nullptr;

cudaEvent_t KernelTimer::take() {
  if (used < pool.size()) return pool[used++];
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
  pool.push_back(e);
  ++used;
  return e;
}

}  // namespace clm

// ===========================================================================
// C ABI
// ===========================================================================
using namespace clm;

extern "C" {

calamanStatus_t calamanCreate(calamanHandle_t *handle) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  *handle = nullptr;
  int dev = 0;
  CLM_CUDA(cudaGetDevice(&dev));
  calamanContext *c = new calamanContext();
  c->device = dev;
  cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, dev);
  const cudaError_t e = cudaMallocHost(&c->h_pinned, 4 * sizeof(double));
  if (e != cudaSuccess) {
    delete c;
    return runtime_status(e);
  }
  *handle = c;
  return ok_status();
}

calamanStatus_t calamanDestroy(calamanHandle_t handle) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (handle->h_pinned) cudaFreeHost(handle->h_pinned);
  for (auto &g : handle->graph)
    if (g.exec) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(g.exec));
  for (auto &g : handle->single)
    if (g.exec) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(g.exec));
  for (auto &g : handle->vjp)
    if (g.exec) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(g.exec));
  if (handle->side) cudaStreamDestroy(handle->side);
  if (handle->side_fork) cudaEventDestroy(handle->side_fork);
  if (handle->side_join) cudaEventDestroy(handle->side_join);
  for (auto &f : handle->lu_fork) f.destroy();
  delete handle;
  return ok_status();
}

calamanStatus_t calamanSetExpmGraphs(calamanHandle_t handle, int enable) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  handle->expm_graphs = enable != 0;
  return ok_status();
}

calamanStatus_t calamanGetExpmGraphs(calamanHandle_t handle, int *enabled, int *cached) {
  if (handle == nullptr || enabled == nullptr || cached == nullptr)
    return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *enabled = handle->expm_graphs;
  *cached = 0;
  for (const auto &g : handle->single) *cached += g.exec != nullptr;
  for (const auto &g : handle->vjp) *cached += g.exec != nullptr;
  return ok_status();
}

calamanStatus_t calamanSetStream(calamanHandle_t handle, calamanStream_t stream) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  handle->stream = static_cast<cudaStream_t>(stream);
  return ok_status();
}

calamanStatus_t calamanGetStream(calamanHandle_t handle, calamanStream_t *stream) {
  if (handle == nullptr || stream == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *stream = handle->stream;
  return ok_status();
}

calamanStatus_t calamanSetPointerMode(calamanHandle_t handle, int mode) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (mode != CALAMAN_POINTER_MODE_HOST && mode != CALAMAN_POINTER_MODE_DEVICE)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  handle->pointer_mode = mode;
  return ok_status();
}

calamanStatus_t calamanGetPointerMode(calamanHandle_t handle, int *mode) {
  if (handle == nullptr || mode == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *mode = handle->pointer_mode;
  return ok_status();
}

const char *calamanGetVersion(void) { return "calaman_b200 0.1.0 (sm_100a)"; }

float calaman_pade_theta_s(int m) { return theta_single(m); }
double calaman_pade_theta_d(int m) { return theta_double(m); }
calamanExpmPlan_t calaman_expm_plan_s(float norm1) { return plan_for<float>(norm1); }
calamanExpmPlan_t calaman_expm_plan_d(double norm1) { return plan_for<double>(norm1); }
int calaman_pade_num_powers(int m) { return pade_coeffs(m) ? pade_num_powers(m) : 0; }
int calaman_pade_num_gemms(int m) { return pade_coeffs(m) ? pade_num_gemms(m) : 0; }

#define CLM_BUFSZ(SUF, T)                                                                     \
  calamanStatus_t calaman_expm_bufferSize_##SUF(calamanSolverHandle_t h, int n, size_t *bytes) { \
    if (n < 1 || bytes == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);          \
    *bytes = expm_bytes<T>(h, n);                                                             \
    return ok_status();                                                                       \
  }                                                                                           \
  calamanStatus_t calaman_pade_bufferSize_##SUF(calamanSolverHandle_t h, int m, int n,        \
                                                size_t *bytes) {                              \
    if (pade_coeffs(m) == nullptr || n < 1 || bytes == nullptr)                               \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                       \
    *bytes = pade_bytes<T>(h, n, m);                                                          \
    return ok_status();                                                                       \
  }
CLM_BUFSZ(s, float)
CLM_BUFSZ(d, double)
CLM_BUFSZ(c, float2)
CLM_BUFSZ(z, double2)
#undef CLM_BUFSZ

calamanStatus_t calaman_expm_s(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int n, const float *A, int lda, float *E, int lde, void *w,
                               size_t lw, int *info, calamanExpmPlan_t *plan) {
  return expm_api<float>(blas, stream, n, A, lda, E, lde, w, lw, info, plan);
}
calamanStatus_t calaman_expm_d(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int n, const double *A, int lda, double *E, int lde, void *w,
                               size_t lw, int *info, calamanExpmPlan_t *plan) {
  return expm_api<double>(blas, stream, n, A, lda, E, lde, w, lw, info, plan);
}
calamanStatus_t calaman_expm_c(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int n, const void *A, int lda, void *E, int lde, void *w, size_t lw,
                               int *info, calamanExpmPlan_t *plan) {
  return expm_api<float2>(blas, stream, n, static_cast<const float2 *>(A), lda,
                          static_cast<float2 *>(E), lde, w, lw, info, plan);
}
calamanStatus_t calaman_expm_z(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int n, const void *A, int lda, void *E, int lde, void *w, size_t lw,
                               int *info, calamanExpmPlan_t *plan) {
  return expm_api<double2>(blas, stream, n, static_cast<const double2 *>(A), lda,
                           static_cast<double2 *>(E), lde, w, lw, info, plan);
}

calamanStatus_t calaman_pade_s(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int m, int n, const float *A, int lda, float *R, int ldr, void *w,
                               size_t lw, int *info) {
  return pade_api<float>(blas, stream, m, n, A, lda, R, ldr, w, lw, info);
}
calamanStatus_t calaman_pade_d(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int m, int n, const double *A, int lda, double *R, int ldr, void *w,
                               size_t lw, int *info) {
  return pade_api<double>(blas, stream, m, n, A, lda, R, ldr, w, lw, info);
}
calamanStatus_t calaman_pade_c(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int m, int n, const void *A, int lda, void *R, int ldr, void *w,
                               size_t lw, int *info) {
  return pade_api<float2>(blas, stream, m, n, static_cast<const float2 *>(A), lda,
                          static_cast<float2 *>(R), ldr, w, lw, info);
}
calamanStatus_t calaman_pade_z(calamanBlasHandle_t blas, calamanSolverHandle_t, calamanStream_t stream,
                               int m, int n, const void *A, int lda, void *R, int ldr, void *w,
                               size_t lw, int *info) {
  return pade_api<double2>(blas, stream, m, n, static_cast<const double2 *>(A), lda,
                           static_cast<double2 *>(R), ldr, w, lw, info);
}

float calaman_matrix_norm1_s(calamanStream_t s, int n, const float *A, int lda, float *cs) {
  return norm1_api<float, float>(s, n, A, lda, cs);
}
double calaman_matrix_norm1_d(calamanStream_t s, int n, const double *A, int lda, double *cs) {
  return norm1_api<double, double>(s, n, A, lda, cs);
}
float calaman_matrix_norm1_c(calamanStream_t s, int n, const void *A, int lda, float *cs) {
  return norm1_api<float2, float>(s, n, static_cast<const float2 *>(A), lda, cs);
}
double calaman_matrix_norm1_z(calamanStream_t s, int n, const void *A, int lda, double *cs) {
  return norm1_api<double2, double>(s, n, static_cast<const double2 *>(A), lda, cs);
}

size_t calaman_horner_bufferSize_s(int n) { return horner_bytes<float>(n); }
size_t calaman_horner_bufferSize_d(int n) { return horner_bytes<double>(n); }
calamanStatus_t calaman_horner_s(calamanBlasHandle_t h, int n, const float *c, int degree,
                                 const float *A, int lda, float *P, int ldp, void *w, size_t wb) {
  return horner_api<float>(h, n, c, degree, A, lda, P, ldp, w, wb);
}
calamanStatus_t calaman_horner_d(calamanBlasHandle_t h, int n, const double *c, int degree,
                                 const double *A, int lda, double *P, int ldp, void *w, size_t wb) {
  return horner_api<double>(h, n, c, degree, A, lda, P, ldp, w, wb);
}

int calaman_paterson_stockmeyer_cost(int degree, int s) { return ps_cost(degree, s); }
int calaman_paterson_stockmeyer_block_size(int degree) { return ps_block_size(degree); }
calamanPatersonStockmeyerPlan_t calaman_paterson_stockmeyer_plan(int degree, int s_requested) {
  return ps_plan(degree, s_requested);
}
size_t calaman_paterson_stockmeyer_power_stride_s(int n) { return ps_stride<float>(n); }
size_t calaman_paterson_stockmeyer_power_stride_d(int n) { return ps_stride<double>(n); }
size_t calaman_paterson_stockmeyer_bufferSize_s(int n, int degree, int s_req) {
  return ps_bytes<float>(n, degree, s_req);
}
size_t calaman_paterson_stockmeyer_bufferSize_d(int n, int degree, int s_req) {
  return ps_bytes<double>(n, degree, s_req);
}
calamanStatus_t calaman_paterson_stockmeyer_s(calamanBlasHandle_t h, int n, const float *c, int degree,
                                              const float *A, int lda, float *P, int ldp, void *w,
                                              size_t wb, int s_req) {
  return ps_api<float>(h, n, c, degree, A, lda, P, ldp, w, wb, s_req);
}
calamanStatus_t calaman_paterson_stockmeyer_d(calamanBlasHandle_t h, int n, const double *c,
                                              int degree, const double *A, int lda, double *P,
                                              int ldp, void *w, size_t wb, int s_req) {
  return ps_api<double>(h, n, c, degree, A, lda, P, ldp, w, wb, s_req);
}

#define CLM_GEMM_API(SUF, T, PT, CPT)                                                          \
  calamanStatus_t calaman_gemm_##SUF(calamanStream_t stream, int m, int n, int k, double alpha, \
                                     CPT A, int lda, CPT B, int ldb, double beta, PT C,         \
                                     int ldc) {                                                 \
    if (m < 0 || n < 0 || k < 0 || lda < (m > 1 ? m : 1) || ldb < (k > 1 ? k : 1) ||            \
        ldc < (m > 1 ? m : 1))                                                                  \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                         \
    if (m == 0 || n == 0) return ok_status();                                                   \
    if (C == nullptr || (k > 0 && (A == nullptr || B == nullptr)))                              \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                         \
    CLM_CUDA(gemm_nn<T>(static_cast<cudaStream_t>(stream), m, n, k, alpha,                      \
                        reinterpret_cast<const T *>(A), lda, reinterpret_cast<const T *>(B),    \
                        ldb, beta, reinterpret_cast<T *>(C), ldc));                             \
    return ok_status();                                                                         \
  }
CLM_GEMM_API(s, float, float *, const float *)
CLM_GEMM_API(d, double, double *, const double *)
CLM_GEMM_API(c, float2, void *, const void *)
CLM_GEMM_API(z, double2, void *, const void *)
#undef CLM_GEMM_API

calamanStatus_t calamanSetDoubleEmulation(calamanHandle_t handle, int digits) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (digits < -1 || digits == 1 || digits > 8) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  handle->fp64_digits = digits;
  return ok_status();
}

calamanStatus_t calamanGetDoubleEmulation(calamanHandle_t handle, int *digits) {
  if (handle == nullptr || digits == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *digits = handle->fp64_digits;
  return ok_status();
}

calamanStatus_t calamanSetFloatSplit(calamanHandle_t handle, int terms) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if (terms != 3 && terms != 6) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  handle->split_terms = terms;
  return ok_status();
}

calamanStatus_t calamanGetFloatSplit(calamanHandle_t handle, int *terms) {
  if (handle == nullptr || terms == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  *terms = handle->split_terms;
  return ok_status();
}

calamanStatus_t calaman_gemm_bf16x_bufferSize(int m, int n, int k, int terms, size_t *bytes) {
  if (m < 1 || n < 1 || k < 1 || (terms != 3 && terms != 6) || bytes == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  *bytes = tc_gemm_workspace_bytes(m, n, k, terms);
  return ok_status();
}

calamanStatus_t calaman_gemm_bf16x_s(calamanStream_t stream, int m, int n, int k, double alpha,
                                     const float *A, int lda, const float *B, int ldb, double beta,
                                     float *C, int ldc, int terms, void *work, size_t work_bytes) {
  if (m < 1 || n < 1 || k < 1 || lda < m || ldb < k || ldc < m || (terms != 3 && terms != 6) ||
      A == nullptr || B == nullptr || C == nullptr || work == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (work_bytes < tc_gemm_workspace_bytes(m, n, k, terms)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  GemmScratch gs;
  gs.ptr = work;
  gs.bytes = work_bytes;
  gs.terms = terms;
  GemmScratchScope gss(&gs);
  CLM_CUDA(gemm_nn<float>(static_cast<cudaStream_t>(stream), m, n, k, alpha, A, lda, B, ldb, beta, C, ldc));
  return ok_status();
}

calamanStatus_t calaman_gemm_ozaki_bufferSize(int m, int n, int k, int is_complex, int digits,
                                              size_t *bytes) {
  if (m < 1 || n < 1 || k < 1 || bytes == nullptr || !oz_gemm_supported(k, is_complex != 0, digits))
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  *bytes = oz_gemm_workspace_bytes(m, n, k, is_complex != 0, digits);
  return ok_status();
}

#define CLM_OZ_API(SUF, T, PT, CPT, CPLX)                                                           \
  calamanStatus_t calaman_gemm_ozaki_##SUF(calamanStream_t stream, int m, int n, int k, double alpha, \
                                          CPT A, int lda, CPT B, int ldb, double beta, PT C, int ldc, \
                                          int digits, void *work, size_t work_bytes) {              \
    if (m < 1 || n < 1 || k < 1 || lda < m || ldb < k || ldc < m || A == nullptr || B == nullptr ||  \
        C == nullptr || work == nullptr || !oz_gemm_supported(k, CPLX, digits))                      \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                             \
    if (work_bytes < oz_gemm_workspace_bytes(m, n, k, CPLX, digits))                                \
      return blas_status(CALAMAN_STATUS_ALLOC_FAILED);                                              \
    CLM_CUDA(oz_gemm<T>(static_cast<cudaStream_t>(stream), m, n, k, alpha,                          \
                        reinterpret_cast<const T *>(A), lda, reinterpret_cast<const T *>(B), ldb,   \
                        beta, reinterpret_cast<T *>(C), ldc, work, work_bytes, digits));            \
    return ok_status();                                                                             \
  }
CLM_OZ_API(d, double, double *, const double *, false)
CLM_OZ_API(z, double2, void *, const void *, true)
#undef CLM_OZ_API

calamanStatus_t calaman_gemm_ozaki_wait_check(calamanStream_t stream, long long spin, void *work,
                                              size_t work_bytes, int *code) {
  constexpr int n = 128;
  const std::size_t ws = oz_gemm_workspace_bytes(n, n, n, false, 2);
  const std::size_t mat = (std::size_t)n * n * sizeof(double);
  if (work == nullptr || code == nullptr || spin < 1) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (work_bytes < align_up(ws, 256) + 3 * mat) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char *w = static_cast<char *>(work);
  double *A = reinterpret_cast<double *>(w + align_up(ws, 256));
  double *B = A + (std::size_t)n * n, *C = B + (std::size_t)n * n;
  CLM_CUDA(cudaMemsetAsync(work, 0, align_up(ws, 256) + 3 * mat, st));
  CLM_CUDA(oz_gemm<double>(st, n, n, n, 1.0, A, n, B, n, 0.0, C, n, work, ws, 2, spin, /*skip_loads=*/1));
  int h = 0;
  CLM_CUDA(cudaMemcpyAsync(&h, work, sizeof(int), cudaMemcpyDeviceToHost, st));
  CLM_CUDA(cudaStreamSynchronize(st));
  *code = h;
  return ok_status();
}

calamanStatus_t calaman_gemm_bf16x_wait_check(calamanStream_t stream, long long spin, void *work, size_t work_bytes,
                                              int *code) {
  constexpr int n = 192, k = 128;  // two k-blocks, ragged tiles
  const std::size_t ws = align_up(tc_gemm_workspace_bytes(n, n, k, 6), 256);
  if (work == nullptr || code == nullptr || spin < 1) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (work_bytes < ws + sizeof(float) * (2 * n * k + n * n)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float *A = reinterpret_cast<float *>(static_cast<char *>(work) + ws), *B = A + n * k, *C = B + n * k;
  CLM_CUDA(cudaMemsetAsync(work, 0, sizeof(int), st));
  CLM_CUDA(tc_gemm_f32(st, n, n, k, 1.0, A, n, B, k, 1.0, C, n, work, ws, 6, spin, /*skip=*/1));
  int h = 0;
  CLM_CUDA(cudaMemcpyAsync(&h, work, sizeof(int), cudaMemcpyDeviceToHost, st));
  CLM_CUDA(cudaStreamSynchronize(st));
  *code = h;
  return ok_status();
}

calamanStatus_t calaman_gemm_bf16x_bufferSize_c(int m, int n, int k, int terms, size_t *bytes) {
  if (m < 1 || n < 1 || k < 1 || (terms != 3 && terms != 6) || bytes == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  *bytes = tc_gemm_workspace_bytes(m, n, k, terms, true);
  return ok_status();
}

calamanStatus_t calaman_gemm_bf16x_c(calamanStream_t stream, int m, int n, int k, double alpha, const void *A,
                                     int lda, const void *B, int ldb, double beta, void *C, int ldc, int terms,
                                     void *work, size_t work_bytes) {
  if (m < 1 || n < 1 || k < 1 || lda < m || ldb < k || ldc < m || (terms != 3 && terms != 6) ||
      A == nullptr || B == nullptr || C == nullptr || work == nullptr)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  if (work_bytes < tc_gemm_workspace_bytes(m, n, k, terms, true)) return blas_status(CALAMAN_STATUS_ALLOC_FAILED);
  GemmScratch gs;
  gs.ptr = work;
  gs.bytes = work_bytes;
  gs.terms = terms;
  GemmScratchScope gss(&gs);
  CLM_CUDA(gemm_nn<float2>(static_cast<cudaStream_t>(stream), m, n, k, alpha, static_cast<const float2 *>(A), lda,
                           static_cast<const float2 *>(B), ldb, beta, static_cast<float2 *>(C), ldc));
  return ok_status();
}

calamanStatus_t calamanSetWorkspace(calamanHandle_t handle, void *d_work, size_t bytes) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  if ((d_work == nullptr) != (bytes == 0) || (reinterpret_cast<std::uintptr_t>(d_work) & 255u) != 0)
    return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  handle->work = d_work;
  handle->work_bytes = bytes;
  return ok_status();
}

size_t calaman_poly_tensor_workspace_s(int n) {
  return n < 1 ? 0 : tc_gemm_workspace_bytes(n, n, n, 6);
}

calamanStatus_t calaman_getrf_bufferSize(int n, size_t *bytes) {
  if (n < 1 || bytes == nullptr) return blas_status(CALAMAN_STATUS_INVALID_VALUE);
  *bytes = lu_scratch_bytes(n);
  return ok_status();
}

#define CLM_LU_API(SUF, T, PT, CPT)                                                            \
  calamanStatus_t calaman_getrf_##SUF(calamanStream_t stream, int n, PT A, int lda,            \
                                      void *scratch, int *d_info) {                            \
    if (n < 1 || n > kMaxDim || lda < n || A == nullptr || scratch == nullptr ||               \
        d_info == nullptr)                                                                     \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                        \
    CLM_CUDA(getrf<T>(static_cast<cudaStream_t>(stream), n, reinterpret_cast<T *>(A), lda,     \
                      scratch, d_info));                                                       \
    return ok_status();                                                                        \
  }                                                                                            \
  calamanStatus_t calaman_getrf_wait_check_##SUF(calamanStream_t stream, int n, PT A, int lda, \
                                                 void *scratch, int drop_from,                 \
                                                 int tries, int *d_info) {                     \
    if (n < 1 || n > kMaxDim || lda < n || A == nullptr || scratch == nullptr ||               \
        drop_from < 0 || tries < 0 || d_info == nullptr)                                       \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                        \
    CLM_CUDA(getrf<T>(static_cast<cudaStream_t>(stream), n, reinterpret_cast<T *>(A), lda,     \
                      scratch, d_info, PanelWait{tries, drop_from}));                          \
    return ok_status();                                                                        \
  }                                                                                            \
  calamanStatus_t calaman_getrs_##SUF(calamanStream_t stream, int n, int nrhs, CPT LU,         \
                                      int lda, const void *scratch, CPT B, int ldb, PT X,      \
                                      int ldx, int *d_info) {                                  \
    if (n < 1 || n > kMaxDim || nrhs < 0 || lda < n || ldb < n || ldx < n || LU == nullptr ||  \
        scratch == nullptr || B == nullptr || X == nullptr || d_info == nullptr)               \
      return blas_status(CALAMAN_STATUS_INVALID_VALUE);                                        \
    CLM_CUDA(getrs<T>(static_cast<cudaStream_t>(stream), n, nrhs,                              \
                      reinterpret_cast<const T *>(LU), lda, scratch,                           \
                      reinterpret_cast<const T *>(B), ldb, reinterpret_cast<T *>(X), ldx,      \
                      d_info));                                                                \
    return ok_status();                                                                        \
  }
CLM_LU_API(s, float, float *, const float *)
CLM_LU_API(d, double, double *, const double *)
CLM_LU_API(c, float2, void *, const void *)
CLM_LU_API(z, double2, void *, const void *)
#undef CLM_LU_API

unsigned long long calamanGetLaunchCount(void) { return g_launch_count(); }

calamanStatus_t calamanSetKernelTiming(calamanHandle_t handle, int enable) {
  if (handle == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  KernelTimer &t = handle->timer;
  t.enabled = enable != 0;
  t.used = 0;
  t.starts.clear();
  t.stops.clear();
  t.flops.clear();
  return ok_status();
}

calamanStatus_t calamanGetKernelTiming(calamanHandle_t handle, calamanKernelTiming_t *out) {
  if (handle == nullptr || out == nullptr) return blas_status(CALAMAN_STATUS_NOT_INITIALIZED);
  KernelTimer &t = handle->timer;
  out->gemm_launches = (long long)t.flops.size();
  out->gemm_ms = 0.0;
  out->gemm_flops = 0.0;
  if (!t.stops.empty()) CLM_CUDA(cudaEventSynchronize(t.stops.back()));
  for (std::size_t i = 0; i < t.flops.size(); ++i) {
    float ms = 0.f;
    CLM_CUDA(cudaEventElapsedTime(&ms, t.starts[i], t.stops[i]));
    out->gemm_ms += ms;
    out->gemm_flops += t.flops[i];
  }
  t.used = 0;
  t.starts.clear();
  t.stops.clear();
  t.flops.clear();
  return ok_status();
}

}  // extern "C"
