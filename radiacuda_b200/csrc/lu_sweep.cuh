// lu_sweep.cuh -- triangular sweeps with the LU factors, one persistent launch
// per factor, and with their transposes.
//
//   sweep_kernel<T, false>    x_k = Linv_k (b_k - sum_{j<k} L_kj x_j)
//   sweep_kernel<T, true>     x_k = Uinv_k (b_k - sum_{j>k} U_kj x_j)
//   sweep_t_kernel<T, false>  x_k = Uinv_k^T (b_k - sum_{j<k} U_jk^T x_j)
//   sweep_t_kernel<T, true>   x_k = Linv_k^T (b_k - sum_{j>k} L_jk^T x_j)
// over blocks of 128.  Each CTA takes the next block in sweep order from a
// counter and streams its tiles of the factor through two register sets while
// the blocks before it are solved.  What bounds a sweep is either the factor's
// bytes or the chain of blocks, so both are kept short:
//   - a solved x_j is its own flag: x starts as a bit pattern that no stored
//     value has (SWEEP_EMPTY), and the 128 threads that need x_j poll its
//     elements themselves: one trip through L2 a block, no fence and no flag
//     after it.  x_{j+1} is asked for while tile j is multiplied; a CTA that
//     is not the next one sleeps in proportion to its distance between polls,
//     or 148 CTAs x 1 KB of polls hold up the one L2 slice they all ask;
//   - products stay in per-lane partial sums over all tiles and are reduced
//     once per block (once per tile, the shuffles held the stream at 1.8 TB/s);
//   - Inv_k and M_k are copied to shared memory when the block is taken;
//   - with FP32 factors and the coupling blocks M_k = Inv_k L_{k,k-1}
//     (Inv_k U_{k,k+1}) everything but the neighbour's part is multiplied by
//     the inverse beforehand, M_k waits in registers in FP64, and after the
//     neighbour's values arrive only x_k = y_k - M_k x_j remains.
// A CTA waits only on blocks taken before its own by CTAs that are running, so
// every wait ends; each is also bounded by `spin` polls, after which the launch
// records an error in *err and every CTA waits for its own copies and returns.
#pragma once

namespace rb {

constexpr int SW_NB = 128, SW_T = 512, SW_W = SW_T / 32, SW_R = SW_NB / SW_W, SW_Q = SW_T / SW_NB, SW_C = SW_NB / SW_Q;
constexpr int SWEEP_SPIN = 1 << 20;  // RADB200_SWEEP_SPIN overrides it (0: a wait runs out at once)
constexpr int SWEEP_NAP = 400, SWEEP_NAP_MAX = 8000;  // ns per block of distance
constexpr unsigned long long SWEEP_EMPTY = ~0ull;

__device__ __forceinline__ void sweep_put(double *p, double v)
{
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (b == SWEEP_EMPTY) b = 0x7ff8000000000000ULL;  // a NaN of another pattern
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}
__device__ __forceinline__ unsigned long long sweep_peek(const double *p)
{
  unsigned long long b;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(p) : "memory");
  return b;
}
// *p (last seen as b) once it is there; bad when the wait ran out
__device__ __forceinline__ double sweep_get(const double *p, unsigned long long b, int dist, int spin, int *err, int *bad)
{
  for (int it = 0; b == SWEEP_EMPTY; it++) {
    if (it > spin || ((it & 255) == 255 && *(volatile int *)err != 0)) {
      atomicExch(err, 1);
      *bad = 1;
      return 0.0;
    }
    if (it > 0 && dist > 2) __nanosleep(min(SWEEP_NAP * (dist - 2), SWEEP_NAP_MAX));
    b = sweep_peek(p);
  }
  return __longlong_as_double((long long)b);
}

// A lane's four columns of a 128-wide row, columns 4 lane ..: zero where the
// row or the column does not exist
template <typename T> struct SweepRow;
template <> struct SweepRow<float> {
  float4 v;
  __device__ __forceinline__ void load(const float *p, bool ok) { v = ok ? __ldcs(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ double get(int c) const { return (double)(c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w); }
};
template <> struct SweepRow<double> {
  double2 a, b;
  __device__ __forceinline__ void load(const double *p, bool ok)
  {
    a = ok ? __ldcs(reinterpret_cast<const double2 *>(p)) : make_double2(0.0, 0.0);
    b = ok ? __ldcs(reinterpret_cast<const double2 *>(p) + 1) : make_double2(0.0, 0.0);
  }
  __device__ __forceinline__ double get(int c) const { return c == 0 ? a.x : c == 1 ? a.y : c == 2 ? b.x : b.y; }
};
// rows of a warp's SW_R per register set
template <typename T> constexpr int sweep_rows() { return sizeof(T) == 4 ? SW_R : SW_R / 2; }
// row pitch of a 128 x 128 block in shared memory: 16 bytes past 128 elements,
// so that 16-byte loads of eight neighbouring rows meet different banks
template <typename T> constexpr int sweep_pitch() { return SW_NB + 16 / (int)sizeof(T); }
template <typename T> constexpr size_t sweep_smem(int blocks) { return (size_t)blocks * SW_NB * sweep_pitch<T>() * sizeof(T); }

// rows 0 .. nb-1 of a 128-wide block to shared memory (cp.async; the caller waits)
template <typename T> __device__ __forceinline__ void sweep_stage(T *dst, const T *src, int nb)
{
  constexpr int E = 16 / sizeof(T), C = SW_NB / E;
  for (int e = threadIdx.x; e < nb * C; e += SW_T) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst + (e / C) * sweep_pitch<T>() + (e % C) * E);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + (size_t)e * E) : "memory");
  }
}
__device__ __forceinline__ void sweep_staged() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T, bool UPPER>
__global__ void __launch_bounds__(SW_T, 1) sweep_kernel(const T *__restrict__ A, int ld, const T *__restrict__ Inv, int n3,
                                                        const double *__restrict__ b, double *x, int *counter, int *err,
                                                        int spin, const T *__restrict__ M)
{
  constexpr int NR = sweep_rows<T>(), NS = SW_R / NR, P = sweep_pitch<T>();
  extern __shared__ __align__(16) unsigned char sweep_dyn[];
  T *sI = reinterpret_cast<T *>(sweep_dyn), *sM = sI + SW_NB * P;  // sM: only with M
  __shared__ double xs[2][SW_NB], as[SW_NB], part[SW_Q][SW_NB];
  __shared__ int s_t, s_bad;
  const int nblk = (n3 + SW_NB - 1) / SW_NB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid & (SW_NB - 1), part_c = tid / SW_NB, c0 = part_c * SW_C;
  if (tid == 0) s_bad = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_t = atomicAdd(counter, 1);
    __syncthreads();
    const int t = s_t;
    if (t >= nblk) return;
    const int k = UPPER ? nblk - 1 - t : t, k0 = k * SW_NB, nb = min(SW_NB, n3 - k0);
    const bool use_m = M != nullptr && t > 0;
    const int tiles = use_m ? t - 1 : t;
    auto col0 = [&](int s) { return (UPPER ? nblk - 1 - s : s) * SW_NB; };
    SweepRow<T> v0[NR], v1[NR];
    auto load = [&](SweepRow<T> *v, int q) {  // set q: rows of tile q / NS
      const int s = q / NS, c = col0(s) + 4 * lane;
#pragma unroll
      for (int i = 0; i < NR; i++) {
        const int row = warp * SW_R + (q % NS) * NR + i;
        v[i].load(A + (size_t)(k0 + row) * ld + c, s < tiles && row < nb && c < ld);
      }
    };
    load(v0, 0);
    sweep_stage(sI, Inv + (size_t)k0 * SW_NB, nb);
    if (use_m) sweep_stage(sM, M + (size_t)k0 * SW_NB, nb);
    unsigned long long seen = SWEEP_EMPTY;
    auto ask = [&](int s) {
      if (tid < SW_NB && s < t && col0(s) + tid < n3) seen = sweep_peek(x + col0(s) + tid);
    };
    // x_j of tile s into xs[s & 1]; false when a wait ran out
    auto arrive = [&](int s) -> bool {
      if (tid < SW_NB) xs[s & 1][tid] = col0(s) + tid < n3 ? sweep_get(x + col0(s) + tid, seen, t - s, spin, err, &s_bad) : 0.0;
      __syncthreads();
      if (s_bad) sweep_staged();  // the launch ends: no copy into shared memory outlives its CTA
      return s_bad == 0;
    };
    double acc[SW_R];
#pragma unroll
    for (int i = 0; i < SW_R; i++) acc[i] = 0.0;
    auto add = [&](const SweepRow<T> *v, int q, double *sum) {
      const double *xp = xs[(q / NS) & 1] + 4 * lane;
      const double x0 = xp[0], x1 = xp[1], x2 = xp[2], x3 = xp[3];
#pragma unroll
      for (int i = 0; i < NR; i++)
        sum[i] += fma(v[i].get(0), x0, fma(v[i].get(1), x1, fma(v[i].get(2), x2, v[i].get(3) * x3)));
    };
    ask(0);
    for (int q = 0; q < tiles * NS; q += 2) {
      load(v1, q + 1);
      if (!arrive(q / NS)) return;
      ask(q / NS + 1);
      add(v0, q, acc);
      if (q + 1 >= tiles * NS) break;
      load(v0, q + 2);
      if (NS == 1) {
        if (!arrive(q + 1)) return;
        ask(q + 2);
      }
      add(v1, q + 1, acc + NR * (NS - 1));
    }
    // b_k minus the products, once across the lanes
#pragma unroll
    for (int i = 0; i < SW_R; i++) {
      double a = acc[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      const int row = warp * SW_R + i;
      if (lane == 0) as[row] = row < nb ? b[k0 + row] - a : 0.0;
    }
    sweep_staged();
    __syncthreads();
    // a quarter of row r times the matching quarter of a vector, then the row
    auto quarter = [&](const T *blk, const double *v) {
      double s0 = 0.0, s1 = 0.0;
      const T *row = blk + r * P + c0;
#pragma unroll
      for (int i = 0; i < SW_C; i += 4) {
        s0 = fma((double)row[i + 1], v[c0 + i + 1], fma((double)row[i], v[c0 + i], s0));
        s1 = fma((double)row[i + 3], v[c0 + i + 3], fma((double)row[i + 2], v[c0 + i + 2], s1));
      }
      return s0 + s1;
    };
    auto whole = [&] { return (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]); };
    if (r < nb) part[part_c][r] = quarter(sI, as);
    __syncthreads();
    double y = tid < nb ? whole() : 0.0;
    if (use_m) {
      double m[SW_C];
#pragma unroll
      for (int i = 0; i < SW_C; i++) m[i] = r < nb ? (double)sM[r * P + c0 + i] : 0.0;
      if (!arrive(t - 1)) return;  // also: everyone is done with part
      const double *xp = xs[(t - 1) & 1] + c0;
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
      for (int i = 0; i < SW_C; i += 4) {
        s0 = fma(m[i], xp[i], s0);
        s1 = fma(m[i + 1], xp[i + 1], s1);
        s2 = fma(m[i + 2], xp[i + 2], s2);
        s3 = fma(m[i + 3], xp[i + 3], s3);
      }
      part[part_c][r] = (s0 + s1) + (s2 + s3);
      __syncthreads();
      if (tid < nb) y -= whole();
    }
    if (tid < nb) sweep_put(x + k0 + tid, y);
  }
}

// LOWER: L^T (backward), else U^T (forward)
template <typename T, bool LOWER>
__global__ void __launch_bounds__(SW_T, 1) sweep_t_kernel(const T *__restrict__ A, int ld, const T *__restrict__ Inv, int n3,
                                                          const double *__restrict__ b, double *x, int *counter, int *err,
                                                          int spin)
{
  constexpr int NR = sweep_rows<T>(), NS = SW_R / NR, P = sweep_pitch<T>();
  extern __shared__ __align__(16) unsigned char sweep_dyn[];
  T *sI = reinterpret_cast<T *>(sweep_dyn);
  __shared__ double xs[2][SW_NB], as[SW_NB], part[SW_Q][SW_NB], red[SW_W][SW_NB];
  __shared__ int s_t, s_bad;
  const int nblk = (n3 + SW_NB - 1) / SW_NB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid & (SW_NB - 1), part_c = tid / SW_NB, c0 = part_c * SW_C;
  if (tid == 0) s_bad = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_t = atomicAdd(counter, 1);
    __syncthreads();
    const int t = s_t;
    if (t >= nblk) return;
    const int k = LOWER ? nblk - 1 - t : t, k0 = k * SW_NB, nb = min(SW_NB, n3 - k0);
    const int col = k0 + 4 * lane;
    auto row0 = [&](int s) { return (LOWER ? nblk - 1 - s : s) * SW_NB; };
    SweepRow<T> v0[NR], v1[NR];
    auto load = [&](SweepRow<T> *v, int q) {
      const int s = q / NS;
#pragma unroll
      for (int i = 0; i < NR; i++) {
        const int row = row0(s) + warp * SW_R + (q % NS) * NR + i;
        v[i].load(A + (size_t)row * ld + col, s < t && row < n3 && col < ld);
      }
    };
    load(v0, 0);
    sweep_stage(sI, Inv + (size_t)k0 * SW_NB, nb);
    unsigned long long seen = SWEEP_EMPTY;
    auto ask = [&](int s) {
      if (tid < SW_NB && s < t && row0(s) + tid < n3) seen = sweep_peek(x + row0(s) + tid);
    };
    auto arrive = [&](int s) -> bool {
      if (tid < SW_NB) xs[s & 1][tid] = row0(s) + tid < n3 ? sweep_get(x + row0(s) + tid, seen, t - s, spin, err, &s_bad) : 0.0;
      __syncthreads();
      if (s_bad) sweep_staged();  // the launch ends: no copy into shared memory outlives its CTA
      return s_bad == 0;
    };
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    auto add = [&](const SweepRow<T> *v, int q) {
      const double *xp = xs[(q / NS) & 1] + warp * SW_R + (q % NS) * NR;
#pragma unroll
      for (int i = 0; i < NR; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[c] = fma(v[i].get(c), xp[i], acc[c]);
    };
    ask(0);
    for (int q = 0; q < t * NS; q += 2) {
      load(v1, q + 1);
      if (!arrive(q / NS)) return;
      ask(q / NS + 1);
      add(v0, q);
      if (q + 1 >= t * NS) break;
      load(v0, q + 2);
      if (NS == 1) {
        if (!arrive(q + 1)) return;
        ask(q + 2);
      }
      add(v1, q + 1);
    }
#pragma unroll
    for (int c = 0; c < 4; c++) red[warp][4 * lane + c] = acc[c];
    __syncthreads();
    if (tid < SW_NB) {
      double a[2] = {tid < nb ? b[k0 + tid] : 0.0, 0.0};
#pragma unroll
      for (int w = 0; w < SW_W; w++) a[w & 1] -= red[w][tid];
      as[tid] = tid < nb ? a[0] + a[1] : 0.0;
    }
    sweep_staged();
    __syncthreads();
    double s0 = 0.0, s1 = 0.0;
    const T *p = sI + c0 * P + r;
#pragma unroll
    for (int i = 0; i < SW_C; i += 2) {
      if (c0 + i < nb) s0 = fma((double)p[i * P], as[c0 + i], s0);
      if (c0 + i + 1 < nb) s1 = fma((double)p[(i + 1) * P], as[c0 + i + 1], s1);
    }
    part[part_c][r] = s0 + s1;
    __syncthreads();
    if (tid < nb) sweep_put(x + k0 + tid, (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]));
  }
}

}  // namespace rb
