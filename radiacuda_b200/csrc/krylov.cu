// krylov.cu -- GMRES (restarted, classical Gram-Schmidt applied twice) on the
// device, and the Newton-Krylov relaxation built on it.
//
// The reference runs GMRES with every dot product round-tripping to the host
// (radgpurlx.cu:2014-2083).  Here an Arnoldi step after the operator is four
// launches and no synchronization: the projections on all basis vectors; the
// update with the second projections in the same pass over the basis; the
// second update with the norm, the new Hessenberg column and its Givens
// rotation (one thread); the normalized new vector.  The last block of each
// launch sums the blocks' partial sums in a fixed order, so the iteration is
// bitwise reproducible.  The host reads one residual estimate per step, and
// where the operator is cheap it has queued the next step's product before
// that.  A step cost up to 10 synchronizations and 25 launches before (up to
// 16 projections per launch): on 9,120 unknowns with an FP64 matrix 0.34 ms,
// of which the matrix takes 0.10 ms from HBM.
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"

namespace rb {


static DBuf g_kpart, g_kscal;

// dots[k] = <V_k, w> for k < nv (chunks of MD_MAX)
static int dots_many(double *const *V, int nv, const double *w, int64_t len, double *out)
{
  for (int s = 0; s < nv; s += MD_MAX) {
    DotSet ds;
    ds.nd = std::min(MD_MAX, nv - s);
    for (int k = 0; k < ds.nd; k++) { ds.a[k] = V[s + k]; ds.b[k] = w; }
    RB_TRY(multidot(ds, len, out + s, g_kpart, g_kscal, 0));
  }
  return 0;
}

// y += sum_k c_k V_k (chunks)
static int axpy_many(double *const *V, const double *c, int nv, int64_t len, double *y)
{
  for (int s = 0; s < nv; s += MD_MAX) {
    AxpySet as;
    as.nv = std::min(MD_MAX, nv - s);
    for (int k = 0; k < as.nv; k++) { as.v[k] = V[s + k]; as.c[k] = c[s + k]; }
    RB_TRY(lincomb(as, len, y, 1, 0));
  }
  return 0;
}

static int vscale(double *v, double a, int64_t len)
{
  AxpySet as; as.nv = 1; as.v[0] = v; as.c[0] = a;
  return lincomb(as, len, v, 0, 0);
}

static int vcopy_axpy(double *y, const double *x, double a, const double *z, double b, int64_t len)
{
  AxpySet as; as.nv = 2; as.v[0] = x; as.c[0] = a; as.v[1] = z; as.c[1] = b;
  return lincomb(as, len, y, 0, 0);
}

// ---- one Arnoldi step ------------------------------------------------------------
constexpr int KR_T = 256, KR_SLICE = 128, KR_MAXV = 201;  // threads, rows per block, basis vectors

// device state of a cycle: Hessenberg columns (rotated), rotations, right-hand side
struct KrView {
  double *part;       // [blocks][KR_MAXV]
  double *h, *h2;     // projections of the step
  double *H;          // [(restart + 1) x restart], row-major
  double *cs, *sn, *g;
  double *inv;        // 1 / |w|
  double *status;     // residual estimate, |w| (copied to the host)
  unsigned *count;    // [3] blocks done, per launch kind
};

// partial dots of this block's rows (in ws) with V_0 .. V_{nv-1}: a warp per vector
__device__ __forceinline__ void slice_dots(const double *V, int ld, int nv, const double *ws, int r0, int rows, double *part)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = warp; k < nv; k += KR_T / 32) {
    const double *v = V + (size_t)k * ld + r0;
    double a = 0.0;
#pragma unroll
    for (int r = lane; r < KR_SLICE; r += 32)
      if (r < rows) a = fma(v[r], ws[r], a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) part[(size_t)blockIdx.x * KR_MAXV + k] = a;
  }
}
__device__ __forceinline__ void sum_parts(const double *part, int nv, double *out)
{
  for (int k = threadIdx.x; k < nv; k += KR_T) {
    double s = 0.0;
#pragma unroll 8
    for (unsigned b = 0; b < gridDim.x; b++) s += __ldcg(part + (size_t)b * KR_MAXV + k);
    out[k] = s;
  }
}
// w slice minus its projections: ws[r] -= sum_k h_k V_k[r], two threads per row
__device__ __forceinline__ void slice_update(const double *V, int ld, int nv, const double *h, double *ws, double *tmp, int r0,
                                             int rows)
{
  __shared__ double hs[KR_MAXV];
  for (int k = threadIdx.x; k < nv; k += KR_T) hs[k] = __ldcg(h + k);
  __syncthreads();
  const int r = threadIdx.x & (KR_SLICE - 1), half = threadIdx.x / KR_SLICE;
  double a = 0.0;
  if (r < rows) {
    const double *v = V + r0 + r;
#pragma unroll 4
    for (int k = half; k < nv; k += KR_T / KR_SLICE) a = fma(hs[k], v[(size_t)k * ld], a);
  }
  if (half) tmp[r] = a;
  __syncthreads();
  if (!half) ws[r] -= a + tmp[r];
  __syncthreads();
}

// h = V^T w
__global__ void __launch_bounds__(KR_T) arnoldi_project_kernel(const double *__restrict__ V, int ld, int n, int nv,
                                                               const double *__restrict__ w, KrView s)
{
  __shared__ double ws[KR_SLICE];
  const int r0 = blockIdx.x * KR_SLICE, rows = min(KR_SLICE, n - r0);
  if (threadIdx.x < KR_SLICE) ws[threadIdx.x] = threadIdx.x < rows ? w[r0 + threadIdx.x] : 0.0;
  __syncthreads();
  slice_dots(V, ld, nv, ws, r0, rows, s.part);
  if (last_block(s.count)) sum_parts(s.part, nv, s.h);
}

// w -= V h, h2 = V^T w
__global__ void __launch_bounds__(KR_T) arnoldi_again_kernel(const double *__restrict__ V, int ld, int n, int nv,
                                                             double *__restrict__ w, KrView s)
{
  __shared__ double ws[KR_SLICE], tmp[KR_SLICE];
  const int r0 = blockIdx.x * KR_SLICE, rows = min(KR_SLICE, n - r0);
  if (threadIdx.x < KR_SLICE) ws[threadIdx.x] = threadIdx.x < rows ? w[r0 + threadIdx.x] : 0.0;
  slice_update(V, ld, nv, s.h, ws, tmp, r0, rows);
  if (threadIdx.x < rows) w[r0 + threadIdx.x] = ws[threadIdx.x];
  slice_dots(V, ld, nv, ws, r0, rows, s.part);
  if (last_block(s.count + 1)) sum_parts(s.part, nv, s.h2);
}

// w -= V h2, |w|; the Hessenberg column j = nv - 1 and its rotation
__global__ void __launch_bounds__(KR_T) arnoldi_finish_kernel(const double *__restrict__ V, int ld, int n, int nv,
                                                              double *__restrict__ w, KrView s, int restart, double bnorm)
{
  __shared__ double ws[KR_SLICE], tmp[KR_SLICE], col[KR_MAXV + 1], c_s[KR_MAXV], s_s[KR_MAXV];
  const int r0 = blockIdx.x * KR_SLICE, rows = min(KR_SLICE, n - r0);
  if (threadIdx.x < KR_SLICE) ws[threadIdx.x] = threadIdx.x < rows ? w[r0 + threadIdx.x] : 0.0;
  slice_update(V, ld, nv, s.h2, ws, tmp, r0, rows);
  if (threadIdx.x < rows) w[r0 + threadIdx.x] = ws[threadIdx.x];
  // |w|^2 of the slice, one warp
  if (threadIdx.x < 32) {
    double a = 0.0;
    for (int r = threadIdx.x; r < rows; r += 32) a = fma(ws[r], ws[r], a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (threadIdx.x == 0) s.part[(size_t)blockIdx.x * KR_MAXV] = a;
  }
  if (!last_block(s.count + 2)) return;
  const int j = nv - 1;
  for (int k = threadIdx.x; k < nv; k += KR_T) {
    col[k] = __ldcg(s.h + k) + __ldcg(s.h2 + k);
    c_s[k] = k < j ? s.cs[k] : 0.0;
    s_s[k] = k < j ? s.sn[k] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double nn = 0.0;
#pragma unroll 8
    for (unsigned b = 0; b < gridDim.x; b++) nn += __ldcg(s.part + (size_t)b * KR_MAXV);
    const double hn = sqrt(nn);
    double a = col[0];
    for (int k = 0; k < j; k++) {
      const double b = col[k + 1];
      col[k] = c_s[k] * a + s_s[k] * b;
      a = -s_s[k] * a + c_s[k] * b;
    }
    const double r = hypot(a, hn);
    const double cj = (r == 0.0) ? 1.0 : a / r, sj = (r == 0.0) ? 0.0 : hn / r, gj = s.g[j];
    col[j] = r;
    s.cs[j] = cj;
    s.sn[j] = sj;
    s.g[j + 1] = -sj * gj;
    s.g[j] = cj * gj;
    s.inv[0] = hn > 0.0 ? 1.0 / hn : 0.0;
    s.status[0] = fabs(sj * gj) / bnorm;
    s.status[1] = hn;
  }
  __syncthreads();
  for (int k = threadIdx.x; k <= j; k += KR_T) s.H[(size_t)k * restart + j] = col[k];
}

// V_{j+1} = w / |w|, and a copy for the operator to work on
__global__ void arnoldi_next_kernel(const double *__restrict__ w, const double *__restrict__ inv, int n,
                                    double *__restrict__ v, double *__restrict__ z)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = w[i] * inv[0];
  v[i] = x;
  z[i] = x;
}

// recorded after a step's status copy
struct StepEvent {
  cudaEvent_t e = nullptr;
  ~StepEvent() { if (e) cudaEventDestroy(e); }
};
// pinned host words for the status of a step (the library is not reentrant)
static double *host_status()
{
  static double *p = nullptr;
  if (!p && cudaMallocHost(&p, 2 * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
  return p;
}

int gmres(Op &op, int n3, int ld, const double *b, double *x, double rtol, int max_iter, int restart, double *relres,
          int *iters, cudaStream_t)
{
  restart = std::max(1, std::min(restart, KR_MAXV - 1));
  const int nb = (n3 + KR_SLICE - 1) / KR_SLICE;
  DBuf Vb, wb, sb;
  RB_TRY(Vb.alloc((size_t)(restart + 1) * ld * sizeof(double)));
  RB_TRY(wb.alloc((size_t)2 * ld * sizeof(double)));
  const size_t words = (size_t)nb * KR_MAXV + 5 * (KR_MAXV + 1) + (size_t)(restart + 1) * restart + 8;
  RB_TRY(sb.alloc(words * sizeof(double)));
  StepEvent ev;
  RB_CUDA(cudaEventCreateWithFlags(&ev.e, cudaEventDisableTiming));
  double *hst = host_status();
  if (!hst) { set_error("pinned host allocation failed"); return RADB200_E_NOMEM; }
  // the matvec reads whole padded rows (ld), so the padding must hold zeros
  RB_CUDA(cudaMemsetAsync(Vb.p, 0, (size_t)(restart + 1) * ld * sizeof(double)));
  RB_CUDA(cudaMemsetAsync(wb.p, 0, (size_t)2 * ld * sizeof(double)));
  RB_CUDA(cudaMemsetAsync(sb.p, 0, words * sizeof(double)));
  KrView kv;
  kv.part = sb.as<double>();
  kv.h = kv.part + (size_t)nb * KR_MAXV;
  kv.h2 = kv.h + KR_MAXV + 1;
  kv.cs = kv.h2 + KR_MAXV + 1;
  kv.sn = kv.cs + KR_MAXV + 1;
  kv.g = kv.sn + KR_MAXV + 1;
  kv.H = kv.g + KR_MAXV + 1;
  kv.inv = kv.H + (size_t)(restart + 1) * restart;
  kv.status = kv.inv + 1;
  kv.count = reinterpret_cast<unsigned *>(kv.status + 2);
  std::vector<double *> V(restart + 1);
  for (int k = 0; k <= restart; k++) V[k] = Vb.as<double>() + (size_t)k * ld;
  double *w = wb.as<double>(), *z = w + ld;
  double bnorm;
  {
    double *bb[1] = {(double *)b};
    RB_TRY(dots_many(bb, 1, b, n3, &bnorm));
    bnorm = sqrt(bnorm);
  }
  if (bnorm == 0.0) bnorm = 1.0;
  int total = 0;
  double rel = 1.0;
  std::vector<double> H((size_t)(restart + 1) * restart), g(restart + 1), y;
  while (true) {
    // r = b - A x
    RB_TRY(op.apply(x, w));
    RB_TRY(vcopy_axpy(V[0], b, 1.0, w, -1.0, n3));
    double beta;
    RB_TRY(dots_many(&V[0], 1, V[0], n3, &beta));
    beta = sqrt(beta);
    rel = beta / bnorm;
    if (!std::isfinite(rel)) { set_error("GMRES: non-finite residual"); return RADB200_E_NUMERIC; }
    if (rel <= rtol || total >= max_iter) break;
    RB_TRY(vscale(V[0], 1.0 / beta, n3));
    RB_CUDA(cudaMemcpyAsync(z, V[0], n3 * sizeof(double), cudaMemcpyDeviceToDevice));
    RB_CUDA(cudaMemcpyAsync(kv.g, &beta, sizeof(double), cudaMemcpyHostToDevice));
    int j = 0;
    bool queued = false;  // the product of step j is already on the stream
    for (; j < restart && total < max_iter; j++, total++) {
      if (!queued) {
        RB_TRY(op.precond(z));
        RB_TRY(op.apply(z, w));
      }
      queued = false;
      arnoldi_project_kernel<<<nb, KR_T>>>(V[0], ld, n3, j + 1, w, kv);
      RB_TRY(check_launch("arnoldi_project_kernel"));
      arnoldi_again_kernel<<<nb, KR_T>>>(V[0], ld, n3, j + 1, w, kv);
      RB_TRY(check_launch("arnoldi_again_kernel"));
      arnoldi_finish_kernel<<<nb, KR_T>>>(V[0], ld, n3, j + 1, w, kv, restart, bnorm);
      RB_TRY(check_launch("arnoldi_finish_kernel"));
      arnoldi_next_kernel<<<(n3 + 255) / 256, 256>>>(w, kv.inv, n3, V[j + 1], z);
      RB_TRY(check_launch("arnoldi_next_kernel"));
      RB_CUDA(cudaMemcpyAsync(hst, kv.status, 2 * sizeof(double), cudaMemcpyDeviceToHost));
      RB_CUDA(cudaEventRecord(ev.e));
      if (op.cheap && j + 1 < restart && total + 1 < max_iter) {
        // the next product runs while the host reads the status; on
        // convergence its result is not used
        RB_TRY(op.apply(z, w));
        queued = true;
      }
      RB_CUDA(cudaEventSynchronize(ev.e));
      if (!std::isfinite(hst[1])) { set_error("GMRES: non-finite residual"); return RADB200_E_NUMERIC; }
      if (hst[0] <= rtol || hst[1] == 0.0) { j++; total++; break; }
    }
    // y = H^-1 g (upper triangular j x j)
    RB_CUDA(cudaMemcpy(H.data(), kv.H, (size_t)j * restart * sizeof(double), cudaMemcpyDeviceToHost));
    RB_CUDA(cudaMemcpy(g.data(), kv.g, (size_t)j * sizeof(double), cudaMemcpyDeviceToHost));
    y.assign(j, 0.0);
    for (int k = j - 1; k >= 0; k--) {
      double s = g[k];
      for (int q = k + 1; q < j; q++) s -= H[(size_t)k * restart + q] * y[q];
      y[k] = s / H[(size_t)k * restart + k];
    }
    RB_CUDA(cudaMemsetAsync(z, 0, n3 * sizeof(double)));
    RB_TRY(axpy_many(V.data(), y.data(), j, n3, z));
    RB_TRY(op.precond(z));
    AxpySet as; as.nv = 1; as.v[0] = z; as.c[0] = 1.0;
    RB_TRY(lincomb(as, n3, x, 1, 0));
  }
  *relres = rel;
  *iters = total;
  return 0;
}

}  // namespace rb
