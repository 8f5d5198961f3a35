// lu.cu -- dense direct solve of the linear-material relaxation system.
//
// No counterpart in the reference (it only iterates, methods 3-11).  For
// linear laws M_i = X_i H_i + Mr_i the fixed point of the relaxation solves
//     A M = X H_ext + Mr,     A = I - X N      (X = block-diagonal chi)
// A is factored in place by a right-looking blocked LU WITHOUT pivoting:
// with the volume-weighted inner product the demagnetization operator -N is
// positive semi-definite, so A is (close to) positive definite and needs no
// row exchanges; a vanishing pivot is reported as RADB200_E_NUMERIC.
//
// Two levels: outer panels of 1536 columns (768 for the last 20,000 rows),
// 128-wide steps inside.  Step k
// (width nb = 128) inside a panel:
//   1. one CTA factors the diagonal block in shared memory (FP64) and writes
//      the inverses of its unit-lower and upper triangles, L_kk^-1 and U_kk^-1
//      (lu_diag.cuh);
//   2. L21 = A21 U_kk^-1 and the panel's U12 = L_kk^-1 A12 as GEMMs (out of
//      place, then copied back), so the triangular solves of the panel also
//      run on the GEMM engine; a narrow update of the panel's other columns,
//      its first 128 rows ahead of the others so that step k+1's diagonal block
//      and U12 run beside them.
// After the panel: its U block row by forward substitution in halves, then one
// trailing update A22 -= L21 U12 with K = the panel width, split into the next panel's
// columns (main stream) and the rest (a side stream, overlapping the next
// panel's factorization).
//   mode F64  : FP64 factors, GEMMs on the FP64 pipe (CUDA cores).
//   mode mixed: FP32 factors, GEMMs on the tcgen05 tensor cores (FP16
//               operands scaled by powers of two, or TF32; FP32 accumulation,
//               gemm_tc.cu), then right-preconditioned FP64 GMRES on A with
//               the FP64 residual (GMRES-IR).
// Triangular solves with the factors use the stored diagonal-block inverses
// (one persistent launch per sweep, lu_sweep.cuh).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include "internal.cuh"
#include "lu_diag.cuh"
#include "lu_sweep.cuh"

namespace rb {

constexpr int LU_NB = 128;  // panel width, also the pitch of the inverse buffers

// A = I - X N, into FP64 or FP32 storage (columns beyond n3 zero)
template <typename T, typename NT>
__global__ void build_A_kernel(const NT *__restrict__ N, const double *__restrict__ mat, int n3, int ld, T *__restrict__ A)
{
  int r = blockIdx.y;
  int e = r / 3, a = r % 3;
  const double *X = mat + (size_t)e * RADB200_MAT_STRIDE;
  double x0 = X[3 * a], x1 = X[3 * a + 1], x2 = X[3 * a + 2];
  const NT *n0 = N + (size_t)(3 * e) * ld;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ld; c += gridDim.x * blockDim.x) {
    double v;
    if (c < n3) v = (r == c ? 1.0 : 0.0) - (x0 * (double)n0[c] + x1 * (double)n0[ld + c] + x2 * (double)n0[2 * (size_t)ld + c]);
    else v = 0.0;
    A[(size_t)r * ld + c] = (T)v;
  }
}

// right-hand side b = X H_ext + Mr
__global__ void build_rhs_kernel(const double *__restrict__ hext, const double *__restrict__ mat, int n, double *__restrict__ b)
{
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double *X = mat + (size_t)e * RADB200_MAT_STRIDE;
  for (int a = 0; a < 3; a++)
    b[3 * e + a] = X[3 * a] * hext[3 * e] + X[3 * a + 1] * hext[3 * e + 1] + X[3 * a + 2] * hext[3 * e + 2] + X[9 + a];
}

// out = x - X y   (A x, given y = N x); transpose != 0: out = x - N^T-side handled by caller
__global__ void apply_A_kernel(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ mat,
                               int n, double *__restrict__ out)
{
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double *X = mat + (size_t)e * RADB200_MAT_STRIDE;
  for (int a = 0; a < 3; a++)
    out[3 * e + a] = x[3 * e + a] - (X[3 * a] * y[3 * e] + X[3 * a + 1] * y[3 * e + 1] + X[3 * a + 2] * y[3 * e + 2]);
}

// ---- diagonal block: factor (unpivoted) and invert both triangles: one CTA,
// blocked by 32 in shared memory (lu_diag.cuh)
static_assert(SW_NB == LU_NB, "the sweeps work on LU_NB blocks");
static_assert(DG_N == LU_NB, "the diagonal-block kernel works on LU_NB x LU_NB blocks");

// ---- CUDA-core GEMM: C[m x n] (=|-=) A[m x k] B[k x n]; 64x64 tile, k-slices of 16
template <typename T>
__global__ void __launch_bounds__(256) gemm_simt_kernel(T *__restrict__ C, int ldc, int m, int n, int k,
                                                        const T *__restrict__ A, int lda, const T *__restrict__ B, int ldb,
                                                        int overwrite)
{
  __shared__ T sA[16][64 + 1];
  __shared__ T sB[16][64 + 1];
  int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  int rb = blockIdx.y * 64, cb = blockIdx.x * 64;
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0;
  for (int kk = 0; kk < k; kk += 16) {
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      int r = e / 16, c = e % 16;
      sA[c][r] = (rb + r < m && kk + c < k) ? A[(size_t)(rb + r) * lda + kk + c] : T(0);
      int kr = e / 64, cc = e % 64;
      sB[kr][cc] = (cb + cc < n && kk + kr < k) ? B[(size_t)(kk + kr) * ldb + cb + cc] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; q++) {
      T a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = sA[q][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = sB[q][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int gr = rb + ty + 16 * i;
    if (gr >= m) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int gc = cb + tx + 16 * j;
      if (gc >= n) continue;
      T *d = C + (size_t)gr * ldc + gc;
      if (overwrite) *d = acc[i][j];
      else *d -= acc[i][j];
    }
  }
}

// dst[r][c] = src[r][c] for r < rows, c < cols (row-major, leading dimensions in elements)
template <typename T>
__global__ void copy2d_kernel(T *__restrict__ dst, int ldd, const T *__restrict__ src, int lds, int rows, int cols)
{
  int64_t tot = (int64_t)rows * cols;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(i / cols), c = (int)(i % cols);
    dst[(size_t)r * ldd + c] = src[(size_t)r * lds + c];
  }
}

// host time spent enqueueing each kind of LU work (RADB200_LU_TIMING=2):
// 0 GEMMs of the panel and U block rows, 1 trailing updates, 2 diagonal blocks, 3 copies
static bool g_lu_host_timing = false;
static double g_lu_host[4];
struct LuHostSpan {
  int i;
  std::chrono::steady_clock::time_point t0;
  explicit LuHostSpan(int k) : i(k)
  {
    if (g_lu_host_timing) t0 = std::chrono::steady_clock::now();
  }
  ~LuHostSpan()
  {
    if (g_lu_host_timing) g_lu_host[i] += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
};

template <typename T>
static int copy2d(T *dst, int ldd, const T *src, int lds, int rows, int cols, cudaStream_t st)
{
  LuHostSpan hs(3);
  int64_t tot = (int64_t)rows * cols;
  int nb = (int)std::min<int64_t>((tot + 255) / 256, 148 * 16);
  copy2d_kernel<T><<<std::max(nb, 1), 256, 0, st>>>(dst, ldd, src, lds, rows, cols);
  return check_launch("copy2d_kernel");
}

template <typename T>
static int gemm(T *C, int ldc, int m, int n, int k, T *A, int lda, const T *B, int ldb, int overwrite, cudaStream_t st,
                int *tc_used, int slot = 0)
{
  if (m <= 0 || n <= 0) return 0;
  LuHostSpan hs(0);
  if (sizeof(T) == 4) {
    int used = 0;
    RB_TRY(tc_gemm_f32((float *)C, ldc, m, n, k, (float *)A, lda, (const float *)B, ldb, st, &used, overwrite, slot));
    if (used) { *tc_used = 1; return 0; }
  }
  dim3 grid((n + 63) / 64, (m + 63) / 64);
  if (grid.y > 65535) { set_error("GEMM grid too large"); return RADB200_E_ARG; }
  gemm_simt_kernel<T><<<grid, 256, 0, st>>>(C, ldc, m, n, k, A, lda, B, ldb, overwrite);
  return check_launch("gemm_simt_kernel");
}

// dst = A B where dst is the same memory as A (c_is_a) or as B: in place on
// the tensor cores when they can (tc_gemm_f32_inplace), else into tmp (pitch
// ldt) and copied back
template <typename T>
static int gemm_to(T *dst, int ldd, int m, int n, int k, T *A, int lda, const T *B, int ldb, bool c_is_a, T *tmp,
                   int ldt, cudaStream_t st, int *tc_used, int slot = 0)
{
  if (m <= 0 || n <= 0) return 0;
  if (sizeof(T) == 4) {
    LuHostSpan hs(0);
    int used = 0;
    RB_TRY(tc_gemm_f32_inplace((float *)dst, ldd, m, n, k, (float *)A, lda, (const float *)B, ldb, st, &used, c_is_a, slot));
    if (used) { *tc_used = 1; return 0; }
  }
  RB_TRY(gemm<T>(tmp, ldt, m, n, k, A, lda, B, ldb, 1, st, tc_used, slot));
  return copy2d<T>(dst, ldd, tmp, ldt, m, n, st);
}

// Optional CUDA-event timing of the trailing updates (A22 -= L21 U12) on the
// stream they are launched on: radb200_update_timing(1) starts collecting,
// radb200_update_stats() returns launches, summed device time, algorithmic
// bytes (C read + written, panels read once) and flops (2 m^2 K) since then.
struct UpdEvents {
  std::vector<cudaEvent_t> ev;
  int used = 0;
  int grow()
  {
    if (2 * used + 2 <= (int)ev.size()) return 0;
    for (int q = 0; q < 512; q++) {
      cudaEvent_t e;
      RB_CUDA(cudaEventCreate(&e));
      ev.push_back(e);
    }
    return 0;
  }
};
static int g_update_timing = 0;
static UpdEvents g_upd_ev;
static double g_upd_bytes = 0.0, g_upd_flops = 0.0;

// Two-level right-looking LU.  Outer panels of LU_OUTER columns; inside a
// panel, 128-wide steps (diagonal block, L21 = A21 U^-1, the panel's own
// U12 = L^-1 A12 and a narrow update of the panel's remaining columns).  The
// panel's U block row for the trailing columns is then solved by block
// forward substitution over its 128-row sub-blocks, and the trailing matrix
// receives ONE update with K = LU_OUTER: the C traffic of the dominant GEMM
// drops by LU_OUTER / 128 against 128-wide steps.
// Outer panel widths: 1536 columns while at least LU_LATE_AT_DEFAULT rows
// remain, then 768.  The trailing GEMMs dominate the early panels (up to K of
// about 1024 they are bound by the traffic of C: 660, 705 and 730 TFLOP/s at
// 1024, 1280 and 1536 columns), the main stream's panel chain the late ones.
// Direct solve of the 60,000^2 system, ms: 1536 then 768 below 20,000 rows 394;
// 1280 then 768 399; 1024 then 768 409 (below 30,000 rows 411); 1536 then 1024
// 400; 1024 throughout 420.  The same rule on 45,000 / 37,500 / 30,000 rows: 157 /
// 108 / 74 (1024 first: 162 / 109 / 74; 768 throughout: 166 / 111 / 74).
constexpr int LU_WIDEST = 2048;  // of all panels
constexpr int LU_OUTER_DEFAULT = 1536, LU_OUTER_LATE_DEFAULT = 768, LU_LATE_AT_DEFAULT = 20000;
// the outer panel width: LU_OUTER_DEFAULT, or RADB200_LU_OUTER (a multiple of
// 128 from 256 to 2048) for tuning; RADB200_LU_OUTER_LATE (same range) is the
// width once fewer than RADB200_LU_LATE_AT rows remain (tuning: the trailing
// GEMMs dominate the early panels, the panel chain the late ones)
static int lu_width_env(const char *name, int dflt)
{
  const char *e = getenv(name);
  int v = e ? atoi(e) : dflt;
  return (v >= 256 && v <= LU_WIDEST && v % LU_NB == 0) ? v : dflt;
}
static int lu_outer()
{
  static int w = 0;
  if (!w) w = lu_width_env("RADB200_LU_OUTER", LU_OUTER_DEFAULT);
  return w;
}
static int lu_outer_at(int remaining)
{
  static int late = 0, at = -1;
  if (!late) {
    late = lu_width_env("RADB200_LU_OUTER_LATE", LU_OUTER_LATE_DEFAULT);
    const char *e = getenv("RADB200_LU_LATE_AT");
    at = e ? std::max(0, atoi(e)) : LU_LATE_AT_DEFAULT;
  }
  return remaining < at ? late : lu_outer();
}

// One-panel look-ahead: the trailing update of outer step k is split into the
// columns of panel k+1 (on the main stream, first) and the rest (on a side
// stream, its grid capped to leave LU_SIDE_FREE_SMS multiprocessors free), so
// that panel k+1 -- its single-CTA diagonal factorizations, narrow GEMMs and
// copies -- is factored on the main stream while the rest of the update runs.
// The main stream waits for the side stream before the U block row of step
// k+1, the only later work that reads or writes the columns the side stream
// updates.  Events order the two streams; nothing waits on the device.
// Inside a panel the first 128 rows of an update go first (rows_first): the
// next diagonal block and its U12 then run on a third stream of high priority
// beside the update of the other rows (the diagonal block is one CTA for 80 us,
// 97 with its launch: 45 ms of the main stream's chain over the 60,000^2
// factorization; 14 left).
constexpr int LU_SIDE_FREE_SMS = 12;  // 60,000^2 direct solve: 8 411, 12 409, 20 407 ms; 28 and 40 slower

struct LuStreams {
  cudaStream_t main = nullptr, side = nullptr, diag = nullptr;
  cudaEvent_t in = nullptr, upd = nullptr, side_done = nullptr, out = nullptr, row = nullptr, diag_done = nullptr;
  int init()
  {
    if (main) return 0;
    RB_CUDA(cudaStreamCreateWithFlags(&main, cudaStreamNonBlocking));
    RB_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    int lo = 0, hi = 0;  // the diagonal block's launches take the next free SM
    RB_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    RB_CUDA(cudaStreamCreateWithPriority(&diag, cudaStreamNonBlocking, hi));
    for (cudaEvent_t *e : {&in, &upd, &side_done, &out, &row, &diag_done}) RB_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    return 0;
  }
};
static LuStreams g_lu_streams;

template <typename T>
static int lu_factor(Intrc &I, T *A, T *Linv, T *Uinv, T *tmp, int *d_err, double tiny, cudaStream_t st, int *tc_used)
{
  const int n3 = I.n3, ld = I.ld;
  T *tmp_row = tmp + std::max((size_t)n3 * LU_NB, (size_t)LU_NB * ld);
  RB_CUDA(cudaFuncSetAttribute(diag_factor_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_SMEM));
  // RADB200_LU_TIMING=1 prints the time of each phase (synchronizes per phase);
  // RADB200_LU_TIMING=2 prints the host's time to enqueue the factorization
  // against its device time (no synchronization inside), which shows whether
  // the launches keep the device fed; RADB200_LU_LOOKAHEAD=0 runs every phase
  // on the caller's stream
  const char *tv = getenv("RADB200_LU_TIMING");
  const int timing_mode = tv ? std::max(1, atoi(tv)) : 0;
  const bool timing = timing_mode == 1;
  cudaEvent_t tq0 = nullptr, tq1 = nullptr;
  auto tq_host = std::chrono::steady_clock::now();
  // RADB200_LU_TIMING=3: events on the main stream between its kinds of work
  // (0 diagonal blocks, 1 L21, 2 U12 in the panel, 3 narrow panel updates,
  // 4 waits for the side stream, 5 U block rows, 6 next panel's update),
  // summed after the factorization: the main stream's critical path by kind
  std::vector<cudaEvent_t> mk_ev;
  std::vector<int> mk_cat;
  if (timing_mode == 2) {
    RB_CUDA(cudaEventCreate(&tq0));
    RB_CUDA(cudaEventCreate(&tq1));
    RB_CUDA(cudaEventRecord(tq0, st));
    tq_host = std::chrono::steady_clock::now();
    g_lu_host_timing = true;
    for (double &h : g_lu_host) h = 0.0;
  }
  const char *la = getenv("RADB200_LU_LOOKAHEAD");
  const bool lookahead = !(la && atoi(la) == 0);
  double tph[4] = {0, 0, 0, 0};
  auto t_last = std::chrono::steady_clock::now();
  auto phase = [&](int p) -> int {
    if (!timing) return 0;
    RB_CUDA(cudaDeviceSynchronize());
    auto t = std::chrono::steady_clock::now();
    tph[p] += std::chrono::duration<double>(t - t_last).count();
    t_last = t;
    return 0;
  };
  cudaStream_t sm = st, ss = st;
  int side_ctas = 0;
  if (lookahead) {
    RB_TRY(g_lu_streams.init());
    sm = g_lu_streams.main;
    ss = g_lu_streams.side;
    RB_CUDA(cudaEventRecord(g_lu_streams.in, st));
    RB_CUDA(cudaStreamWaitEvent(sm, g_lu_streams.in, 0));
    RB_CUDA(cudaStreamWaitEvent(ss, g_lu_streams.in, 0));
    int dev = 0, nsm = 0;
    RB_CUDA(cudaGetDevice(&dev));
    RB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const char *fs = getenv("RADB200_LU_FREE_SMS");  // tuning override
    side_ctas = std::max(1, nsm - ((fs && atoi(fs) > 0) ? atoi(fs) : LU_SIDE_FREE_SMS));
  }
  auto mark = [&](int cat) -> int {
    if (timing_mode != 3) return 0;
    cudaEvent_t e;
    RB_CUDA(cudaEventCreate(&e));
    RB_CUDA(cudaEventRecord(e, sm));
    mk_ev.push_back(e);
    mk_cat.push_back(cat);
    return 0;
  };
  bool side_pending = false, ahead = false;
  auto at = [&](int r, int c) { return A + (size_t)r * ld + c; };
  // C[m x n] -= A B with the update's timing events on stream q
  auto update = [&](T *C, int m, int n, int k, T *Ap, const T *Bp, cudaStream_t q, int slot, int cap) -> int {
    if (m <= 0 || n <= 0) return 0;
    LuHostSpan hs(1);
    if (g_update_timing) {
      RB_TRY(g_upd_ev.grow());
      RB_CUDA(cudaEventRecord(g_upd_ev.ev[2 * g_upd_ev.used], q));
    }
    int used = 0;
    if (sizeof(T) == 4) {
      RB_TRY(tc_gemm_f32((float *)C, ld, m, n, k, (float *)Ap, ld, (const float *)Bp, ld, q, &used, 0, slot, cap));
      if (used) *tc_used = 1;
    }
    if (!used) RB_TRY(gemm<T>(C, ld, m, n, k, Ap, ld, Bp, ld, 0, q, tc_used));
    if (g_update_timing) {
      RB_CUDA(cudaEventRecord(g_upd_ev.ev[2 * g_upd_ev.used + 1], q));
      g_upd_ev.used++;
      // algorithmic bytes: C read + written, the L and U panels read once (as
      // FP16 copies when the tensor cores took FP16 operands)
      const double opb = used == 2 ? 2.0 : (double)sizeof(T);
      g_upd_bytes += (double)sizeof(T) * 2.0 * m * n + opb * ((double)m * k + (double)k * n);
      g_upd_flops += 2.0 * m * n * k;
    }
    return 0;
  };
  auto diag = [&](int j0, int jb, cudaStream_t q) -> int {
    LuHostSpan hs(2);
    diag_factor_kernel<T><<<1, DG_T, DG_SMEM, q>>>(A, ld, j0, jb, Linv, Uinv, d_err, tiny);
    return check_launch("diag_factor_kernel");
  };
  // U12 of step j0 inside its panel: L_jj^-1 A12 (out of place: tmp_row)
  auto u12 = [&](int j0, int pend, cudaStream_t q, int slot) -> int {
    const int jb = std::min(LU_NB, pend - j0), rest = j0 + jb, w = pend - rest;
    return w <= 0 ? 0
                  : gemm_to<T>(at(j0, rest), ld, jb, w, jb, Linv + (size_t)j0 * LU_NB, LU_NB, at(j0, rest), ld, false,
                               tmp_row, LU_WIDEST, q, tc_used, slot);
  };
  // An update of the rows from r0 on of a panel that ends at column pend:
  // run(r, rows) first for the next step's 128 rows, whose diagonal block and
  // U12 then go on beside run() of the others
  auto rows_first = [&](int r0, int pend, auto run) -> int {
    const int rows = n3 - r0, first = std::min(LU_NB, rows);
    if (!lookahead) return run(r0, rows);
    RB_TRY(run(r0, first));
    RB_CUDA(cudaEventRecord(g_lu_streams.row, sm));
    RB_CUDA(cudaStreamWaitEvent(g_lu_streams.diag, g_lu_streams.row, 0));
    RB_TRY(diag(r0, std::min(LU_NB, pend - r0), g_lu_streams.diag));
    RB_TRY(u12(r0, pend, g_lu_streams.diag, 2));
    RB_CUDA(cudaEventRecord(g_lu_streams.diag_done, g_lu_streams.diag));
    ahead = true;
    return rows > first ? run(r0 + first, rows - first) : 0;
  };
  // U rows r0 .. r1 of the n columns from c0 on by halves: the upper half, its
  // product off the lower half, the lower half.  Every level reads and
  // converts half of the rows once (row by row of blocks, the rows above were
  // converted again for each: 3,584 instead of 1,536 rows per 1024).
  auto urows = [&](auto self, int r0, int r1, int c0, int n) -> int {
    const int blocks = (r1 - r0 + LU_NB - 1) / LU_NB, mid = std::min(r1, r0 + (blocks + 1) / 2 * LU_NB);
    if (blocks == 1)
      return gemm_to<T>(at(r0, c0), ld, r1 - r0, n, r1 - r0, Linv + (size_t)r0 * LU_NB, LU_NB, at(r0, c0), ld, false, tmp, ld,
                        sm, tc_used);
    RB_TRY(self(self, r0, mid, c0, n));
    RB_TRY(gemm<T>(at(mid, c0), ld, r1 - mid, n, mid - r0, at(mid, r0), ld, at(r0, c0), ld, 0, sm, tc_used));
    return self(self, mid, r1, c0, n);
  };
  for (int K0 = 0, NBe = 0; K0 < n3; K0 += NBe) {
    NBe = std::min(lu_outer_at(n3 - K0), n3 - K0);
    const int pend = K0 + NBe;  // end of the panel's columns
    // ---- factor the panel columns [K0, pend) over rows [K0, n3) (main stream;
    // the previous step updated these columns there first)
    for (int j0 = K0; j0 < pend; j0 += LU_NB) {
      const int jb = std::min(LU_NB, pend - j0), rest = j0 + jb, m = n3 - rest, w = pend - rest;
      const bool done = ahead;  // the diagonal block and the panel's U12 of this step
      if (ahead) {
        RB_CUDA(cudaStreamWaitEvent(sm, g_lu_streams.diag_done, 0));
        ahead = false;
      } else {
        RB_TRY(diag(j0, jb, sm));
      }
      RB_TRY(mark(0));
      RB_TRY(phase(0));
      if (m <= 0) break;
      // L21 = A21 U_jj^-1   (tmp: m x LU_NB)
      RB_TRY(gemm_to<T>(at(rest, j0), ld, m, jb, jb, at(rest, j0), ld, Uinv + (size_t)j0 * LU_NB, LU_NB, true, tmp, LU_NB,
                        sm, tc_used));
      RB_TRY(mark(1));
      if (w > 0) {
        if (!done) RB_TRY(u12(j0, pend, sm, 0));
        RB_TRY(mark(2));
        // narrow update of the panel: A[rest:, rest:pend] -= L21 U12
        RB_TRY(rows_first(rest, pend, [&](int r, int mr) -> int {
          return gemm<T>(at(r, rest), ld, mr, w, jb, at(r, j0), ld, at(j0, rest), ld, 0, sm, tc_used);
        }));
        RB_TRY(mark(3));
      }
      RB_TRY(phase(1));
    }
    const int T0 = pend, mT = n3 - pend;
    if (mT <= 0) break;
    // the columns right of this panel must carry the previous step's update
    if (side_pending) {
      RB_CUDA(cudaEventRecord(g_lu_streams.side_done, ss));
      RB_CUDA(cudaStreamWaitEvent(sm, g_lu_streams.side_done, 0));
      side_pending = false;
    }
    RB_TRY(mark(4));
    // ---- U block row of the trailing columns: forward substitution with the
    // panel's unit-lower diagonal block
    RB_TRY(urows(urows, K0, pend, T0, mT));
    RB_TRY(mark(5));
    RB_TRY(phase(2));
    // ---- trailing update A22 -= L21 U12 with K = NBe: the next panel's
    // columns on the main stream, the rest on the side stream
    const int nxt = lookahead ? std::min(lu_outer_at(mT), mT) : mT;  // the next panel's width
    RB_TRY(rows_first(T0, T0 + nxt, [&](int r, int mr) -> int {
      return update(at(r, T0), mr, nxt, NBe, at(r, K0), at(K0, T0), sm, 0, 0);
    }));
    RB_TRY(mark(6));
    if (mT > nxt) {
      RB_CUDA(cudaEventRecord(g_lu_streams.upd, sm));
      RB_CUDA(cudaStreamWaitEvent(ss, g_lu_streams.upd, 0));
      RB_TRY(update(at(T0, T0 + nxt), mT, mT - nxt, NBe, at(T0, K0), at(K0, T0 + nxt), ss, 1, side_ctas));
      side_pending = true;
    }
    RB_TRY(phase(3));
  }
  if (lookahead) {
    if (ahead) RB_CUDA(cudaStreamWaitEvent(sm, g_lu_streams.diag_done, 0));
    RB_CUDA(cudaEventRecord(g_lu_streams.side_done, ss));
    RB_CUDA(cudaStreamWaitEvent(sm, g_lu_streams.side_done, 0));
    RB_CUDA(cudaEventRecord(g_lu_streams.out, sm));
    RB_CUDA(cudaStreamWaitEvent(st, g_lu_streams.out, 0));
  }
  if (timing)
    fprintf(stderr, "[radb200 LU n=%d %s] diag %.3f s, panel %.3f s, U block rows %.3f s, trailing %.3f s\n", n3,
            sizeof(T) == 4 ? "fp32" : "fp64", tph[0], tph[1], tph[2], tph[3]);
  if (timing_mode == 3 && !mk_ev.empty()) {
    RB_CUDA(cudaEventSynchronize(mk_ev.back()));
    double cat[7] = {0, 0, 0, 0, 0, 0, 0};
    for (size_t i = 1; i < mk_ev.size(); i++) {
      float ms = 0.f;
      RB_CUDA(cudaEventElapsedTime(&ms, mk_ev[i - 1], mk_ev[i]));
      cat[mk_cat[i]] += 1e-3 * ms;
    }
    for (cudaEvent_t e : mk_ev) cudaEventDestroy(e);
    fprintf(stderr,
            "[radb200 LU n=%d %s] main stream: diagonal blocks %.4f s, L21 %.4f s, panel U12 %.4f s, narrow updates "
            "%.4f s, waits for the side stream %.4f s, U block rows %.4f s, next panel's update %.4f s\n",
            n3, sizeof(T) == 4 ? "fp32" : "fp64", cat[0], cat[1], cat[2], cat[3], cat[4], cat[5], cat[6]);
  }
  if (timing_mode == 2) {
    const double host = std::chrono::duration<double>(std::chrono::steady_clock::now() - tq_host).count();
    RB_CUDA(cudaEventRecord(tq1, st));
    RB_CUDA(cudaEventSynchronize(tq1));
    float ms = 0.f;
    RB_CUDA(cudaEventElapsedTime(&ms, tq0, tq1));
    fprintf(stderr,
            "[radb200 LU n=%d %s] host enqueue %.3f s (panel GEMMs %.3f, trailing updates %.3f, diagonal blocks %.3f, "
            "copies %.3f), device %.3f s\n",
            n3, sizeof(T) == 4 ? "fp32" : "fp64", host, g_lu_host[0], g_lu_host[1], g_lu_host[2], g_lu_host[3], 1e-3 * ms);
    g_lu_host_timing = false;
    cudaEventDestroy(tq0);
    cudaEventDestroy(tq1);
  }
  return 0;
}

// Coupling blocks of FP32 factors for the sweeps: Mf[k] = Linv_k L_{k,k-1}
// (k >= 1) and Mb[k] = Uinv_k U_{k,k+1} (k < nblk - 1), 128 x 128 each, rows
// beyond block k's size and columns beyond its neighbour's zero.  With them a
// sweep finishes block k as x_k = y_k - M_k x_j once x_j of the block before
// it (in sweep order) appears, y_k = Inv_k (b_k - the other products) having
// been formed while waiting.  One CTA per block and direction, FP32 products
// of 128 terms, 8 x 8 outputs per thread.
__global__ void __launch_bounds__(256) sweep_m_kernel(const float *__restrict__ A, int ld, const float *__restrict__ Linv,
                                                      const float *__restrict__ Uinv, int n3, float *__restrict__ Mf,
                                                      float *__restrict__ Mb)
{
  __shared__ float sI[LU_NB][33];      // 32 columns of the inverse
  __shared__ float sB[32][LU_NB + 4];  // the matching 32 rows of the coupling block
  const int nblk = (n3 + LU_NB - 1) / LU_NB;
  const int k = blockIdx.x >> 1, upper = blockIdx.x & 1;
  if (upper ? k >= nblk - 1 : k < 1) return;
  const int k0 = k * LU_NB, nb = min(LU_NB, n3 - k0);
  const int j0 = (upper ? k + 1 : k - 1) * LU_NB, nbj = min(LU_NB, n3 - j0);
  const float *Inv = (upper ? Uinv : Linv) + (size_t)k0 * LU_NB;
  float *out = (upper ? Mb : Mf) + (size_t)k * LU_NB * LU_NB;
  const int tr = threadIdx.x / 16, tc = threadIdx.x % 16;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int c = 0; c < 8; c++) acc[i][c] = 0.f;
  for (int q0 = 0; q0 < LU_NB; q0 += 32) {
    for (int e = threadIdx.x; e < LU_NB * 32; e += 256) {
      const int r = e / 32, q = e % 32;
      sI[r][q] = r < nb ? Inv[(size_t)r * LU_NB + q0 + q] : 0.f;
      const int qr = e / LU_NB, c = e % LU_NB;
      sB[qr][c] = (q0 + qr < nb && c < nbj) ? A[(size_t)(k0 + q0 + qr) * ld + j0 + c] : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int q = 0; q < 32; q++) {
      float a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] = sI[tr * 8 + i][q];
#pragma unroll
      for (int c = 0; c < 8; c++) b[c] = sB[q][tc * 8 + c];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int c = 0; c < 8; c++) acc[i][c] = fmaf(a[i], b[c], acc[i][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int c = 0; c < 8; c++) out[(size_t)(tr * 8 + i) * LU_NB + tc * 8 + c] = acc[i][c];
}

static DBuf g_tri_err;  // error flag of the sweeps

// error flag of the sweeps: 0, or 1 when a wait ran out (then cleared)
int tri_sweep_error(int *flag)
{
  *flag = 0;
  if (!g_tri_err.p) return 0;
  RB_CUDA(cudaMemcpy(flag, g_tri_err.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (*flag) RB_CUDA(cudaMemset(g_tri_err.p, 0, sizeof(int)));
  return 0;
}

// Buffers of the sweeps for the current factors (also factors that came with a
// restored state): two vectors, two counters; FP32 factors: coupling blocks.
static int sweep_prepare(Intrc &I, int mode)
{
  RB_TRY(I.tri_sync.alloc(2 * (size_t)I.ld * sizeof(double) + 2 * sizeof(int)));
  if (!g_tri_err.p) {
    RB_TRY(g_tri_err.alloc(sizeof(int)));
    RB_CUDA(cudaMemset(g_tri_err.p, 0, sizeof(int)));
  }
  if (mode == RADB200_LU_TF32 && !I.sweep_m.p && I.n3 > LU_NB) {
    const int nblk = (I.n3 + LU_NB - 1) / LU_NB;
    RB_TRY(I.sweep_m.alloc(2 * (size_t)nblk * LU_NB * LU_NB * sizeof(float)));
    const float *inv = I.LUinv.as<float>();
    float *Mf = I.sweep_m.as<float>(), *Mb = Mf + (size_t)nblk * LU_NB * LU_NB;
    sweep_m_kernel<<<2 * nblk, 256>>>(I.LU32.as<float>(), I.ld, inv, inv + (size_t)I.n3 * LU_NB, I.n3, Mf, Mb);
    RB_TRY(check_launch("sweep_m_kernel"));
  }
  return 0;
}

template <typename T> static int sweeps(Intrc &I, const T *A, int transposed, double *x, cudaStream_t st)
{
  const int n3 = I.n3, ld = I.ld, nblk = (n3 + LU_NB - 1) / LU_NB;
  double *y = I.tri_sync.as<double>(), *z = y + ld;
  int *count = reinterpret_cast<int *>(z + ld), *err = g_tri_err.as<int>();
  const T *L = I.LUinv.as<T>(), *U = L + (size_t)n3 * LU_NB;
  RB_CUDA(cudaMemsetAsync(y, 0xff, 2 * (size_t)ld * sizeof(double), st));  // SWEEP_EMPTY
  RB_CUDA(cudaMemsetAsync(count, 0, 2 * sizeof(int), st));
  int dev = 0, nsm = 0;
  RB_CUDA(cudaGetDevice(&dev));
  RB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int grid = std::min(nblk, nsm);
  const char *e = getenv("RADB200_SWEEP_SPIN");
  const int spin = e ? std::min(std::max(atoi(e), 0), SWEEP_SPIN) : SWEEP_SPIN;
  auto run = [&](auto kernel, int blocks, auto... args) -> int {
    const size_t smem = sweep_smem<T>(blocks);
    RB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, SW_T, smem, st>>>(args...);
    return check_launch("sweep_kernel");
  };
  if (transposed) {
    RB_TRY(run(sweep_t_kernel<T, false>, 1, A, ld, U, n3, x, y, count, err, spin));
    RB_TRY(run(sweep_t_kernel<T, true>, 1, A, ld, L, n3, y, z, count + 1, err, spin));
  } else {
    // (FP64 factors: no coupling blocks)
    const T *Mf = sizeof(T) == 4 ? I.sweep_m.as<T>() : nullptr, *Mb = Mf ? Mf + (size_t)nblk * LU_NB * LU_NB : nullptr;
    RB_TRY(run(sweep_kernel<T, false>, Mf ? 2 : 1, A, ld, L, n3, x, y, count, err, spin, Mf));
    RB_TRY(run(sweep_kernel<T, true>, Mf ? 2 : 1, A, ld, U, n3, y, z, count + 1, err, spin, Mb));
  }
  RB_CUDA(cudaMemcpyAsync(x, z, (size_t)n3 * sizeof(double), cudaMemcpyDeviceToDevice, st));
  return 0;
}

// x <- A^-1 x (or A^-T x) with the kept factors
static int lu_apply(Intrc &I, int transposed, double *x, cudaStream_t st)
{
  if (I.lu_mode != RADB200_LU_F64 && I.lu_mode != RADB200_LU_TF32) {
    set_error("no LU factors on this interaction");
    return RADB200_E_ARG;
  }
  RB_TRY(sweep_prepare(I, I.lu_mode));
  return I.lu_mode == RADB200_LU_F64 ? sweeps<double>(I, I.LU64.as<double>(), transposed, x, st)
                                     : sweeps<float>(I, I.LU32.as<float>(), transposed, x, st);
}

int lu_precond(Intrc &I, double *x, cudaStream_t st) { return lu_apply(I, 0, x, st); }

// x <- A^-T x with the kept factors (the adjoint's preconditioner)
int lu_precond_transposed(Intrc &I, double *x, cudaStream_t st) { return lu_apply(I, 1, x, st); }

struct LinOp : Op {
  Intrc &I;
  double *tmp;
  double t_mv = 0.0, t_pc = 0.0;  // seconds in products / sweeps (RADB200_TIMING only)
  LinOp(Intrc &i, double *t) : I(i), tmp(t) {}
  int apply(const double *v, double *out) override
  {
    const double t0 = timing_on() ? (cudaDeviceSynchronize(), now_s()) : 0.0;
    RB_TRY(run_matvec(I, v, nullptr, 1.0, tmp, 0));
    apply_A_kernel<<<(I.n + 127) / 128, 128>>>(v, tmp, I.mat.as<double>(), I.n, out);
    RB_TRY(check_launch("apply_A_kernel"));
    if (t0 > 0.0) { cudaDeviceSynchronize(); t_mv += now_s() - t0; }
    return 0;
  }
  int precond(double *v) override
  {
    const double t0 = timing_on() ? (cudaDeviceSynchronize(), now_s()) : 0.0;
    RB_TRY(lu_precond(I, v, 0));
    if (t0 > 0.0) { cudaDeviceSynchronize(); t_pc += now_s() - t0; }
    return 0;
  }
};

int lu_build(Intrc &I, int mode, double *factor_seconds)
{
  if (I.lu_mode == mode && !I.lu_of_d) { *factor_seconds = 0.0; return 0; }
  return lu_build_x(I, mode, I.mat.as<double>(), 0, factor_seconds);
}

// max |A_ii| (as float bits: non-negative floats order like their bits)
template <typename T>
__global__ void diag_absmax_kernel(const T *__restrict__ A, int ld, int n3, unsigned *__restrict__ out)
{
  float m = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x)
    m = fmaxf(m, (float)fabs((double)A[(size_t)i * ld + i]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

template <typename T>
__global__ void add_diag_kernel(T *__restrict__ A, int ld, int n3, double sigma)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) A[(size_t)i * ld + i] = (T)((double)A[(size_t)i * ld + i] + sigma);
}

// Pivots at or below LU_TINY of the largest |A_ii| stop the unpivoted
// factorization; it is then redone on A + sigma I, sigma = LU_SHIFT of that
// scale (at least LU_SHIFT), and the FP64 GMRES that refines every solve --
// always with the unshifted operator -- takes the shifted factors as its
// preconditioner.  For physical materials (chi >= 0) A is diagonally similar
// to a symmetric positive-definite matrix, so every leading minor is positive
// and the shift is never needed; it covers unphysical inputs (a negative
// susceptibility that zeroes a self block) and rounding.
constexpr double LU_TINY = 1e-12, LU_SHIFT = 1e-3;

int lu_build_x(Intrc &I, int mode, const double *X, int of_d, double *factor_seconds)
{
  auto t0 = std::chrono::steady_clock::now();
  const int n3 = I.n3, ld = I.ld;
  I.lu_mode = -1;
  DBuf err;  // [pivot flag, max |A_ii| as float bits]
  dim3 bgrid((ld + 255) / 256 > 64 ? 64 : (ld + 255) / 256, n3);
  int tc_used = 0;
  size_t es = (mode == RADB200_LU_F64) ? sizeof(double) : sizeof(float);
  RB_TRY(I.LUinv.alloc(2 * (size_t)n3 * LU_NB * es));
  RB_TRY(I.lu_scratch.alloc((std::max((size_t)n3 * LU_NB, (size_t)LU_NB * ld) + LU_NB * LU_WIDEST) * es));
  if (mode == RADB200_LU_F64) {
    I.LU32.release();
    RB_TRY(I.LU64.alloc((size_t)n3 * ld * sizeof(double)));
  } else {
    I.LU64.release();
    RB_TRY(I.LU32.alloc((size_t)n3 * ld * sizeof(float)));
  }
  RB_TRY(err.alloc(2 * sizeof(int)));
  double tiny = 0.0;
  I.lu_shift = 0.0;
  int herr = 0, tcflag = 0;
  for (int attempt = 0; attempt < 2; attempt++) {
    RB_CUDA(cudaMemset(err.p, 0, 2 * sizeof(int)));
    unsigned *mx = reinterpret_cast<unsigned *>(err.as<int>() + 1);
    const int nb = std::min((n3 + 255) / 256, 148 * 4);
    if (mode == RADB200_LU_F64) {
      if (I.N64.p) build_A_kernel<double, double><<<bgrid, 256>>>(I.N64.as<double>(), X, n3, ld, I.LU64.as<double>());
      else build_A_kernel<double, float><<<bgrid, 256>>>(I.N32.as<float>(), X, n3, ld, I.LU64.as<double>());
      RB_TRY(check_launch("build_A_kernel"));
      if (attempt) add_diag_kernel<double><<<(n3 + 255) / 256, 256>>>(I.LU64.as<double>(), ld, n3, I.lu_shift);
      else diag_absmax_kernel<double><<<nb, 256>>>(I.LU64.as<double>(), ld, n3, mx);
    } else {
      if (I.N64.p) build_A_kernel<float, double><<<bgrid, 256>>>(I.N64.as<double>(), X, n3, ld, I.LU32.as<float>());
      else build_A_kernel<float, float><<<bgrid, 256>>>(I.N32.as<float>(), X, n3, ld, I.LU32.as<float>());
      RB_TRY(check_launch("build_A_kernel"));
      if (attempt) add_diag_kernel<float><<<(n3 + 255) / 256, 256>>>(I.LU32.as<float>(), ld, n3, I.lu_shift);
      else diag_absmax_kernel<float><<<nb, 256>>>(I.LU32.as<float>(), ld, n3, mx);
    }
    RB_TRY(check_launch(attempt ? "add_diag_kernel" : "diag_absmax_kernel"));
    if (!attempt) {
      unsigned bits = 0;
      RB_CUDA(cudaMemcpy(&bits, mx, sizeof(unsigned), cudaMemcpyDeviceToHost));
      float scale = 0.f;
      memcpy(&scale, &bits, sizeof(float));
      tiny = LU_TINY * (double)scale;
      if (!(tiny > 1e-300)) tiny = 1e-300;
    }
    if (mode == RADB200_LU_F64) {
      double *inv = I.LUinv.as<double>();
      RB_TRY(lu_factor<double>(I, I.LU64.as<double>(), inv, inv + (size_t)n3 * LU_NB, I.lu_scratch.as<double>(),
                               err.as<int>(), tiny, 0, &tc_used));
    } else {
      float *inv = I.LUinv.as<float>();
      RB_TRY(lu_factor<float>(I, I.LU32.as<float>(), inv, inv + (size_t)n3 * LU_NB, I.lu_scratch.as<float>(),
                              err.as<int>(), tiny, 0, &tc_used));
    }
    RB_CUDA(cudaMemcpy(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost));
    RB_TRY(tc_error_flag(&tcflag));
    if (tcflag) { I.lu_mode = -1; set_error("LU: a tensor-core update timed out waiting for its MMAs"); return RADB200_E_TIMEOUT; }
    if (!herr) break;
    I.lu_shift = LU_SHIFT * std::max(1.0, tiny / LU_TINY);
    if (timing_on())
      fprintf(stderr, "RADB200_TIMING LU: pivot at or below %.3e; refactoring A + %.3e I\n", tiny, I.lu_shift);
  }
  if (herr) {
    I.lu_mode = -1;
    I.lu_shift = 0.0;
    set_error("LU: vanishing pivot (A and A + sigma I not factorable without pivoting)");
    return RADB200_E_NUMERIC;
  }
  I.sweep_m.release();
  RB_TRY(sweep_prepare(I, mode));
  I.lu_mode = mode;
  I.lu_of_d = of_d;
  I.lu_solve_id = I.solve_id;
  I.lu_tc = tc_used;
  RB_CUDA(cudaDeviceSynchronize());
  *factor_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return 0;
}

int direct_solve(Intrc &I, int mode, double rtol, int max_iter, double *status)
{
  auto t0 = std::chrono::steady_clock::now();
  const int n3 = I.n3, ld = I.ld;
  double tf = 0.0;
  PhaseClock pc;
  RB_TRY(lu_build(I, mode, &tf));
  pc.mark("solve: factors");
  RB_TRY(I.work.alloc((size_t)4 * ld * sizeof(double)));
  double *b = I.work.as<double>(), *tmp = b + ld;
  RB_CUDA(cudaMemset(I.work.p, 0, (size_t)4 * ld * sizeof(double)));
  build_rhs_kernel<<<(I.n + 127) / 128, 128>>>(I.hext.as<double>(), I.mat.as<double>(), I.n, b);
  RB_TRY(check_launch("build_rhs_kernel"));
  RB_CUDA(cudaMemcpy(I.M.p, b, n3 * sizeof(double), cudaMemcpyDeviceToDevice));
  RB_TRY(lu_precond(I, I.M.as<double>(), 0));
  LinOp op(I, tmp);
  double relres = 0.0;
  int its = 0;
  const int rc = gmres(op, n3, ld, b, I.M.as<double>(), rtol, max_iter, 30, &relres, &its, 0);
  // a sweep that gave up leaves NaN, so its flag is read (and cleared) whatever gmres said
  int tri_err = 0;
  RB_TRY(tri_sweep_error(&tri_err));
  if (tri_err) { set_error("direct solve: a triangular sweep timed out waiting for a block"); return RADB200_E_TIMEOUT; }
  RB_TRY(rc);
  RB_CUDA(cudaDeviceSynchronize());
  if (timing_on())
    fprintf(stderr, "RADB200_TIMING solve: refinement, %d its: products %.3f ms, sweeps %.3f ms\n", its, 1e3 * op.t_mv,
            1e3 * op.t_pc);
  pc.mark("solve: refinement");
  status[0] = relres;
  status[1] = its;
  status[2] = tf;
  status[3] = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return 0;
}

}  // namespace rb

extern "C" RADB200_API int radb200_update_timing(int on)
{
  rb::g_update_timing = on;
  rb::g_upd_ev.used = 0;
  rb::g_upd_bytes = 0.0;
  rb::g_upd_flops = 0.0;
  return 0;
}

extern "C" RADB200_API int radb200_update_stats(int64_t *launches, double *seconds, double *bytes, double *flops)
{
  RB_CUDA(cudaDeviceSynchronize());
  double ms_total = 0.0;
  for (int i = 0; i < rb::g_upd_ev.used; i++) {
    float ms = 0.f;
    RB_CUDA(cudaEventElapsedTime(&ms, rb::g_upd_ev.ev[2 * i], rb::g_upd_ev.ev[2 * i + 1]));
    ms_total += ms;
  }
  *launches = rb::g_upd_ev.used;
  *seconds = 1e-3 * ms_total;
  *bytes = rb::g_upd_bytes;
  *flops = rb::g_upd_flops;
  return 0;
}
