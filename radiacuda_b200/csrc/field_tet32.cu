// field_tet32.cu -- field of an all-tetrahedron model with FP32 terms.
//
// The vertex/edge form of tet_fast (formulas.cuh): vertex offsets formed in
// FP64 and rounded to FP32; distances, edge integrals and solid angles in
// FP32; weights and sums in FP64.  Bound by instruction issue: the library's
// log1pf, atan2f, division and square root made 793 thread-instructions a
// pair, this form 377 (8,000 tetrahedra, 1e6 points: 223 ms before, 126 ms).
// Most pairs are distant, and there each element is short:
//   L / 2 = artanh(x),   x = l / (Ra + Rb) <= 1/6:    a quotient, 3 terms;
//   half solid angle = arctan(num / den) <= 0.025:     a quotient, 2 terms,
// when the point is at least 4 times the longest edge from vertex 0 (every
// distance is then at least 3 of them).  The quotients' corrections, and what
// rounding took from Ra + Rb, go into the last addition of each.
// In a smooth body the terms of an inner edge cancel among its tetrahedra, if
// all take the same value for it.  So an edge distant by itself (Ra + Rb >= 6 l)
// takes the distant form in every tetrahedron, also in those that are not.
// 2-norm and largest error at a point of B against FP64, the body of chi = 1000
// relaxed, 20,000 tetrahedra, 1e6 points: 3.2e-8, 6.2e-7 (the library's form
// 4.0e-8, 7.6e-7; by whole tetrahedra, without this rule, 6.9e-8, 2.1e-6);
// 3,000 tetrahedra 3.4e-8 (3.8e-8; 6.4e-8).
// Nearer pairs take the log1pf and atan2f forms.  A warp pays for the longer
// path when any of its lanes needs it, so larger point sets are first put in
// Morton order; each point's sum runs over the tetrahedra in their own order
// either way.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>

#include "internal.cuh"

namespace rb {

namespace {

constexpr int T32_TILE = 32, T32_T = 256;
constexpr int T32_D = 66;  // doubles per unit: v (12), 2 C a_f (12), 2 C g_e (18), point map (12), field map (9), M (3)
constexpr int T32_F = 20;  // floats per unit: edge lengths (6), face normals m (12), (4 longest edge)^2, 1 if both maps are diagonal
constexpr int T32_REC = T32_D * 8 + T32_F * 4;  // bytes of a unit's record: the doubles, then the floats
static_assert(T32_REC % 16 == 0 && (T32_D * 8) % 16 == 0, "records are copied 16 bytes at a time");

__device__ __forceinline__ float rcp32(float d)
{
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return y;
}
// n / d = q + c: the product with the approximate reciprocal and its Newton
// correction, which the caller adds last, in the same rounding as its series;
// t is what d is short of its unrounded value by
__device__ __forceinline__ float quot32(float n, float d, float t, float &c)
{
  const float y = rcp32(d), q = n * y;
  c = fmaf(-q, t, fmaf(-d, q, n)) * y;
  return q;
}
// sqrt by the approximate reciprocal root and one Newton correction
__device__ __forceinline__ float root32(float s)
{
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
  const float g = s * y;
  return fmaf(0.5f * y, fmaf(-g, g, s), g);
}

// half the edge integral, artanh(l / (Ra + Rb)), for Ra + Rb >= 6 l
__device__ __forceinline__ float far_half_L(float ra, float rb, float l)
{
  const float s = ra + rb;
  float c;  // ra and rb differ by less than a factor 2: (ra - s) + rb is exact
  const float x = quot32(l, s, (ra - s) + rb, c), z = x * x;
  // artanh(x) = x (1 + z p(z)), least maximum error 2.3e-9 for z <= 1/36
  const float p = fmaf(fmaf(0.1477081972f, z, 0.1999480270f), z, 0.3333334154f);
  return x + fmaf(x * z, p, c);
}

struct D3 {
  double x, y, z;
};

// one pair: acc += its B or H in the lab frame
__device__ __forceinline__ void tet32_pair(const double *__restrict__ sd, const float *__restrict__ sf, D3 P, int what,
                                           double *acc)
{
  const double *T = sd + 42, *F = sd + 54;
  const bool diag = sf[19] != 0.f;
  const double dx = P.x - T[9], dy = P.y - T[10], dz = P.z - T[11];
  double qx, qy, qz;
  if (diag) {
    qx = T[0] * dx;
    qy = T[4] * dy;
    qz = T[8] * dz;
  } else {
    qx = T[0] * dx + T[1] * dy + T[2] * dz;
    qy = T[3] * dx + T[4] * dy + T[5] * dz;
    qz = T[6] * dx + T[7] * dy + T[8] * dz;
  }
  float rx[4], ry[4], rz[4], R[4], d[6];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    rx[k] = (float)(sd[3 * k] - qx);
    ry[k] = (float)(sd[3 * k + 1] - qy);
    rz[k] = (float)(sd[3 * k + 2] - qz);
    R[k] = fmaf(rx[k], rx[k], fmaf(ry[k], ry[k], rz[k] * rz[k]));
  }
  const bool far = R[0] >= sf[18];
#pragma unroll
  for (int e = 0; e < 6; e++) {
    const int a = tet_edge_a(e), b = tet_edge_b(e);
    d[e] = fmaf(rx[a], rx[b], fmaf(ry[a], ry[b], rz[a] * rz[b]));
  }
  double h0 = 0.0, h1 = 0.0, h2 = 0.0;
  bool inside = false;
  auto edge_add = [&](int e, float half_L) {
    const double L = (double)half_L;
    h0 = fma(L, sd[24 + 3 * e], h0);
    h1 = fma(L, sd[25 + 3 * e], h1);
    h2 = fma(L, sd[26 + 3 * e], h2);
  };
  auto face_add = [&](int f, float half_omega) {
    const double w = (double)half_omega;
    h0 = fma(w, sd[12 + 3 * f], h0);
    h1 = fma(w, sd[13 + 3 * f], h1);
    h2 = fma(w, sd[14 + 3 * f], h2);
  };
  if (far) {
#pragma unroll
    for (int k = 0; k < 4; k++) R[k] = root32(R[k]);
#pragma unroll
    for (int e = 0; e < 6; e++) edge_add(e, far_half_L(R[tet_edge_a(e)], R[tet_edge_b(e)], sf[e]));
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const int a = tet_face_a(f), b = tet_face_b(f), c = tet_face_c(f);
      const float num = fmaf(rx[a], sf[6 + 3 * f], fmaf(ry[a], sf[7 + 3 * f], rz[a] * sf[8 + 3 * f]));
      const float den = fmaf(fmaf(R[a], R[b], d[tet_pair(a, b)]), R[c], fmaf(d[tet_pair(a, c)], R[b], d[tet_pair(b, c)] * R[a]));
      float cw;
      const float w = quot32(-num, den, 0.f, cw), u = w * w;
      // arctan(w) = w (1 + u p(u)), least maximum error 3e-11 for u <= 0.0012
      face_add(f, w + fmaf(w * u, fmaf(0.1998287159f, u, -0.3333333076f), cw));
    }
  } else {
    float Q[4];  // the distances as the distant form takes them
#pragma unroll
    for (int k = 0; k < 4; k++) {
      Q[k] = root32(R[k]);
      R[k] = sqrtf(R[k]);
    }
#pragma unroll
    for (int e = 0; e < 6; e++) {
      const int a = tet_edge_a(e), b = tet_edge_b(e);
      const float l = sf[e];
      // an edge distant by itself takes the form that it takes in every other tetrahedron
      if (Q[a] + Q[b] >= 6.f * l) edge_add(e, far_half_L(Q[a], Q[b], l));
      else edge_add(e, 0.5f * edge_L(rx[a], ry[a], rz[a], R[a], rx[b], ry[b], rz[b], R[b], d[e], l));
    }
    double total = 0.0;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const int a = tet_face_a(f), b = tet_face_b(f), c = tet_face_c(f);
      const float num = rx[a] * sf[6 + 3 * f] + ry[a] * sf[7 + 3 * f] + rz[a] * sf[8 + 3 * f];
      const float den = R[a] * R[b] * R[c] + d[tet_pair(a, b)] * R[c] + d[tet_pair(a, c)] * R[b] + d[tet_pair(b, c)] * R[a];
      const float w = atan2f(-num, den);
      total += (double)w;
      face_add(f, w);
    }
    inside = total < -3.141592653589793;
  }
  if (what == 2) h0 = h1 = h2 = 0.0;
  if (what != 1 && inside) {
    h0 += sd[63];
    h1 += sd[64];
    h2 += sd[65];
  }
  if (diag) {
    acc[0] = fma(F[0], h0, acc[0]);
    acc[1] = fma(F[4], h1, acc[1]);
    acc[2] = fma(F[8], h2, acc[2]);
  } else {
    acc[0] += F[0] * h0 + F[1] * h1 + F[2] * h2;
    acc[1] += F[3] * h0 + F[4] * h1 + F[5] * h2;
    acc[2] += F[6] * h0 + F[7] * h1 + F[8] * h2;
  }
}

// the records of units [ub, ub + nu)
__global__ void tet32_record_kernel(GeomView g, int ub, int nu, unsigned char *__restrict__ rec)
{
  const int64_t tot = (int64_t)nu * (T32_D + T32_F);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(e / (T32_D + T32_F)), f = (int)(e - (int64_t)k * (T32_D + T32_F));
    const int4 un = g.units[ub + k];  // {kind, polyhedron, transform, diagonal point map}
    const double *t = g.tetrec + (size_t)g.tetidx[un.y] * TET_REC_FIELD, *T = g.trf + (size_t)un.z * RADB200_TRF_STRIDE;
    unsigned char *o = rec + (size_t)k * T32_REC;
    if (f < T32_D) {
      const double C2 = 2.0 / (4.0 * 3.141592653589793238);
      double v;
      if (f < 12) v = t[f];
      else if (f < 42) v = C2 * t[18 + f];  // a_f from 30, g_e from 42
      else if (f < 63) v = T[f - 42];
      else v = g.poly[(size_t)un.y * RADB200_POLY_STRIDE + 3 + (f - 63)];
      reinterpret_cast<double *>(o)[f] = v;
    } else {
      const int q = f - T32_D;
      float v;
      if (q < 18) v = (float)t[12 + q];  // lengths, then normals
      else if (q == 18) {
        double m = 0.0;
        for (int c = 0; c < 6; c++) m = fmax(m, t[12 + c]);
        v = (float)(16.0 * m * m);
      } else {
        const double *F = T + 12;
        v = un.w && F[1] == 0.0 && F[2] == 0.0 && F[3] == 0.0 && F[5] == 0.0 && F[6] == 0.0 && F[7] == 0.0 ? 1.f : 0.f;
      }
      reinterpret_cast<float *>(o + T32_D * 8)[q] = v;
    }
  }
}

// perm: the order of the points (null: as they are).  Records come in through
// two shared buffers, the next tile's copy under way while a tile is summed.
__global__ void __launch_bounds__(T32_T) field_tet32_kernel(const unsigned char *__restrict__ rec,
                                                            const double *__restrict__ pts, int64_t npts,
                                                            const unsigned *__restrict__ perm, int what,
                                                            double *__restrict__ out, int nu, int chunk, int accumulate)
{
  __shared__ __align__(16) unsigned char buf[2][T32_TILE * T32_REC];
  const int tid = threadIdx.x;
  const int u0 = blockIdx.y * chunk, u1 = min(nu, u0 + chunk);
  const int64_t i = (int64_t)blockIdx.x * T32_T + tid;
  const int64_t idx = i < npts ? (perm ? (int64_t)perm[i] : i) : -1;
  D3 P{0, 0, 0};
  if (idx >= 0) P = D3{pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2]};
  double acc[3] = {0, 0, 0};
  auto fetch = [&](int base, int b) {
    const int n16 = min(T32_TILE, u1 - base) * (T32_REC / 16);
    const unsigned char *src = rec + (size_t)base * T32_REC;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(buf[b]);
    for (int e = tid; e < n16; e += T32_T)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + 16 * (size_t)e) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(u0, 0);
  for (int base = u0, b = 0; base < u1; base += T32_TILE, b ^= 1) {
    if (base + T32_TILE < u1) {
      fetch(base + T32_TILE, b ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int cnt = min(T32_TILE, u1 - base);
    for (int k = 0; k < cnt; k++) {
      const unsigned char *r = buf[b] + k * T32_REC;
      tet32_pair(reinterpret_cast<const double *>(r), reinterpret_cast<const float *>(r + T32_D * 8), P, what, acc);
    }
    __syncthreads();  // before the tile after next is copied over this one
  }
  if (idx >= 0) {
    double *o = out + ((size_t)blockIdx.y * npts + idx) * 3;
#pragma unroll
    for (int c = 0; c < 3; c++) o[c] = accumulate ? o[c] + acc[c] : acc[c];
  }
}

// floats in an order that unsigned integers share
__device__ __forceinline__ unsigned ordered(float x)
{
  const unsigned u = __float_as_uint(x);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float unordered(unsigned u)
{
  return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

// box[0..2] the smallest, box[3..5] the largest coordinates (ordered bits)
__global__ void point_box_kernel(const double *__restrict__ pts, int64_t n, unsigned *__restrict__ box)
{
  unsigned lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0, 0, 0};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    for (int c = 0; c < 3; c++) {
      const float x = (float)pts[3 * i + c];
      if (!isfinite(x)) continue;
      lo[c] = min(lo[c], ordered(x));
      hi[c] = max(hi[c], ordered(x));
    }
  for (int c = 0; c < 3; c++) {
    lo[c] = __reduce_min_sync(0xffffffffu, lo[c]);
    hi[c] = __reduce_max_sync(0xffffffffu, hi[c]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(box + c, lo[c]);
      atomicMax(box + 3 + c, hi[c]);
    }
  }
}

__device__ __forceinline__ unsigned spread3(unsigned x)
{
  x = (x | (x << 16)) & 0x030000FF;
  x = (x | (x << 8)) & 0x0300F00F;
  x = (x | (x << 4)) & 0x030C30C3;
  return (x | (x << 2)) & 0x09249249;
}

__global__ void point_key_kernel(const double *__restrict__ pts, int64_t n, const unsigned *__restrict__ box,
                                 unsigned *__restrict__ key, unsigned *__restrict__ idx)
{
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float ext = 0.f, lo[3];
  for (int c = 0; c < 3; c++) {
    lo[c] = unordered(box[c]);
    ext = fmaxf(ext, unordered(box[3 + c]) - lo[c]);
  }
  unsigned k = 0;
  for (int c = 0; c < 3; c++) {
    const float t = ((float)pts[3 * i + c] - lo[c]) / ext * 1023.f;
    k |= spread3(t > 0.f ? min((unsigned)t, 1023u) : 0u) << c;  // NaN: 0
  }
  key[i] = k;
  idx[i] = (unsigned)i;
}

__global__ void tet32_reduce_kernel(const double *__restrict__ part, int nc, int64_t n3, double *__restrict__ out, int accumulate)
{
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  double s = accumulate ? out[i] : 0.0;
  for (int c = 0; c < nc; c++) s += part[(size_t)c * n3 + i];
  out[i] = s;
}

// The Morton order of the points into perm.buf; scratch from the block pool
struct PointOrder {
  DBuf box, key, key2, idx, idx2, tmp;
  const unsigned *perm = nullptr;
  int build(const double *d_pts, int64_t n, cudaStream_t st)
  {
    const unsigned init[6] = {~0u, ~0u, ~0u, 0, 0, 0};
    RB_TRY(box.upload(init, sizeof(init)));
    for (DBuf *b : {&key, &key2, &idx, &idx2}) RB_TRY(b->alloc((size_t)n * sizeof(unsigned)));
    point_box_kernel<<<148 * 2, 256, 0, st>>>(d_pts, n, box.as<unsigned>());
    RB_TRY(check_launch("point_box_kernel"));
    point_key_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_pts, n, box.as<unsigned>(), key.as<unsigned>(),
                                                                  idx.as<unsigned>());
    RB_TRY(check_launch("point_key_kernel"));
    size_t bytes = 0;
    RB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, key.as<unsigned>(), key2.as<unsigned>(), idx.as<unsigned>(),
                                            idx2.as<unsigned>(), (int)n, 0, 30, st));
    RB_TRY(tmp.alloc(bytes));
    RB_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, bytes, key.as<unsigned>(), key2.as<unsigned>(), idx.as<unsigned>(),
                                            idx2.as<unsigned>(), (int)n, 0, 30, st));
    perm = idx2.as<unsigned>();
    return 0;
  }
};

}  // namespace

int launch_tet32_field(const GeomView &g, const double *d_pts, int64_t npts, int what, double *d_out, int ub, int ue,
                       int accumulate, DBuf &scratch, cudaStream_t st)
{
  PointOrder order;
  if (npts >= T32_SORT_MIN && npts <= INT32_MAX) RB_TRY(order.build(d_pts, npts, st));
  const int64_t nblk = (npts + T32_T - 1) / T32_T;
  const int nu = ue - ub;
  DBuf rec;
  RB_TRY(rec.alloc((size_t)nu * T32_REC));
  const int rblk = (int)std::min<int64_t>(((int64_t)nu * (T32_D + T32_F) + 255) / 256, 148 * 8);
  tet32_record_kernel<<<rblk, 256, 0, st>>>(g, ub, nu, rec.as<unsigned char>());
  RB_TRY(check_launch("tet32_record_kernel"));
  // too few points for the GPU: split the tetrahedra as well
  const int64_t target = 148 * 8;
  int nchunk = nblk < target ? (int)((target + nblk - 1) / nblk) : 1;
  nchunk = std::min(std::min(nchunk, nu), 65535);
  const int chunk = (nu + nchunk - 1) / nchunk;
  nchunk = (nu + chunk - 1) / chunk;
  double *dst = d_out;
  if (nchunk > 1) {
    RB_TRY(scratch.alloc((size_t)nchunk * npts * 3 * sizeof(double)));
    dst = scratch.as<double>();
  }
  field_tet32_kernel<<<dim3((unsigned)nblk, (unsigned)nchunk), T32_T, 0, st>>>(rec.as<unsigned char>(), d_pts, npts, order.perm,
                                                                              what, dst, nu, chunk, nchunk > 1 ? 0 : accumulate);
  RB_TRY(check_launch("field_tet32_kernel"));
  if (nchunk == 1) return 0;
  const int64_t n3 = npts * 3;
  tet32_reduce_kernel<<<(unsigned)((n3 + 255) / 256), 256, 0, st>>>(scratch.as<double>(), nchunk, n3, d_out, accumulate);
  return check_launch("tet32_reduce_kernel");
}

}  // namespace rb
