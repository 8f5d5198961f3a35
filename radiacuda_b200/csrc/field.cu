// field.cu -- B / H / M at observation points from all field sources.
//
// Replaces radGPU_FldKernelT + radGPU_FldRecMagKernel + their partial-sum
// reductions (reference radgpu_fld.cu:381-553, 788-909) and the host coil
// loop (radgpu_fld.cpp:542-617).  Design:
//   - one thread per observation point, FP64 accumulation in registers;
//   - every thread of a CTA walks the same (source, image) unit list, so the
//     source records are warp-uniform loads served by L1 broadcast -- no
//     shared-memory staging is needed because each record feeds hundreds of
//     transcendental operations;
//   - symmetry / orientation images are applied in-kernel (point mapped into
//     the source's own frame, field mapped back with s*M);
//   - coils (arc currents, current cuboids) and background fields run on the
//     device with the magnets;
//   - when there are too few points to fill the GPU, the unit list is split
//     over gridDim.y chunks whose partial sums land in a scratch buffer and
//     are added in a fixed order (bitwise reproducible).
#include <cooperative_groups.h>

#include <algorithm>

#include "internal.cuh"

namespace rb {

// KIND: 0 cuboid, 1 polyhedron (face-by-face form), 2 polyhedron (vertex/edge
// form where available), 3 arc current, 4 background.  One kernel is compiled
// per kind so each gets the register budget of its own formula.
enum { UK_REC = 0, UK_POLY = 1, UK_POLY_FAST = 2, UK_ARC = 3, UK_BKG = 4, UK_TET = 5, UK_TRI = 6 };

template <typename T, int KIND>
__device__ __forceinline__ V3<double> eval_unit(const GeomView &g, int4 u, V3<double> P, int what)
{
  const double *Tr = g.trf + (size_t)u.z * RADB200_TRF_STRIDE;
  // point in the source's own frame: q = M^-1 (P - V)
  double dx = P.x - __ldg(Tr + 9), dy = P.y - __ldg(Tr + 10), dz = P.z - __ldg(Tr + 11);
  V3<double> q;
  if (u.w) q = mk3<double>(__ldg(Tr + 0) * dx, __ldg(Tr + 4) * dy, __ldg(Tr + 8) * dz);  // diagonal (identity, mirrors)
  else
    q = mk3<double>(__ldg(Tr + 0) * dx + __ldg(Tr + 1) * dy + __ldg(Tr + 2) * dz,
                    __ldg(Tr + 3) * dx + __ldg(Tr + 4) * dy + __ldg(Tr + 5) * dz,
                    __ldg(Tr + 6) * dx + __ldg(Tr + 7) * dy + __ldg(Tr + 8) * dz);
  V3<double> f = mk3<double>(0, 0, 0);
  if (KIND == UK_REC) {
    const double *r = g.rec + (size_t)u.y * RADB200_REC_STRIDE;
    double jx = __ldg(r + 9), jy = __ldg(r + 10), jz = __ldg(r + 11);
    V3<double> qc = mk3<double>(q.x - __ldg(r + 0), q.y - __ldg(r + 1), q.z - __ldg(r + 2));
    V3<double> hd = mk3<double>(0.5 * __ldg(r + 3), 0.5 * __ldg(r + 4), 0.5 * __ldg(r + 5));
    if (jx != 0.0 || jy != 0.0 || jz != 0.0) {
      if (what != 2) f = cuboid_J(qc, hd, mk3<double>(jx, jy, jz), g.g);
    } else {
      double mx = __ldg(r + 6), my = __ldg(r + 7), mz = __ldg(r + 8);
      if (what == 2) {
        int in = (fabs(qc.x) < hd.x) && (fabs(qc.y) < hd.y) && (fabs(qc.z) < hd.z);
        if (in) f = mk3<double>(mx, my, mz);
      } else {
        // cuboids stay FP64 in every precision mode, as in the reference (its
        // cuboid kernel radgpu_fld.cu:788-882 has no FP32 variant)
        V3<double> Tt, Ss;
        int in = cuboid_TS(qc, hd, g.g, Tt, Ss);
        const double cx = CUBOID_C * mx, cy = CUBOID_C * my, cz = CUBOID_C * mz;
        f = mk3<double>(Tt.x * cx - Ss.z * cy - Ss.y * cz, -Ss.z * cx + Tt.y * cy - Ss.x * cz,
                        -Ss.y * cx - Ss.x * cy + Tt.z * cz);
        if (what == 0 && in) { f.x += mx; f.y += my; f.z += mz; }
      }
    }
  } else if (KIND == UK_POLY_FAST && __ldg(&g.tp.tinfo[u.y].y) >= 0) {
    // vertex/edge form (formulas.cuh: tet_fast for tetrahedra, poly_fast otherwise)
    const double *pr = g.poly + (size_t)u.y * RADB200_POLY_STRIDE;
    double h[3];
    int ti = __ldg(g.tetidx + u.y);
    int in = (ti >= 0) ? tet_fast<T, false>(g.tetrec + (size_t)ti * TET_REC_FIELD, q, h) : poly_fast<T, false>(g.tp, u.y, q, h);
    if (what == 2) f = in ? mk3<double>(__ldg(pr + 3), __ldg(pr + 4), __ldg(pr + 5)) : mk3<double>(0, 0, 0);
    else {
      f = mk3<double>(h[0], h[1], h[2]);
      if (what == 0 && in) { f.x += __ldg(pr + 3); f.y += __ldg(pr + 4); f.z += __ldg(pr + 5); }
    }
  } else if (KIND == UK_POLY || KIND == UK_POLY_FAST) {
    const double *pr = g.poly + (size_t)u.y * RADB200_POLY_STRIDE;
    double mx = __ldg(pr + 3), my = __ldg(pr + 4), mz = __ldg(pr + 5);
    int f0 = __ldg(g.poly_info + 4 * u.y), nf = __ldg(g.poly_info + 4 * u.y + 1);
    // the reference's polygon face form uses this 15-digit pi (radplnr2.cpp:32)
    const double CH = 1.0 / (4.0 * 3.14159265358979);
    int inside = 1;
    double hx = 0, hy = 0, hz = 0;
    for (int fi = f0; fi < f0 + nf; fi++) {
      const double *R = g.face + (size_t)fi * RADB200_FACE_STRIDE;
      double r0 = __ldg(R + 0), r1 = __ldg(R + 1), r2 = __ldg(R + 2), r3 = __ldg(R + 3), r4 = __ldg(R + 4),
             r5 = __ldg(R + 5), r6 = __ldg(R + 6), r7 = __ldg(R + 7), r8 = __ldg(R + 8), cz = __ldg(R + 9);
      // local normal component of M (row 2 of R)
      double mloc = r6 * mx + r7 * my + r8 * mz;
      int v0 = __ldg(g.face_vtx + 2 * fi), nv = __ldg(g.face_vtx + 2 * fi + 1);
      const double *vt = g.vtx2d + 2 * (size_t)v0;
      double plx = r0 * q.x + r1 * q.y + r2 * q.z, ply = r3 * q.x + r4 * q.y + r5 * q.z, plz = r6 * q.x + r7 * q.y + r8 * q.z;
      double s0, s1, s2;
      int in = polygon_S(vt, g.edge + EDGE_REC * (size_t)v0, nv, cz, mk3<double>(plx, ply, plz), g.g, s0, s1, s2);
      if (!in) inside = 0;
      if (what != 2) {
        double w = -CH * mloc;
        // H_obj += R^T (w S)
        hx += w * (r0 * s0 + r3 * s1 + r6 * s2);
        hy += w * (r1 * s0 + r4 * s1 + r7 * s2);
        hz += w * (r2 * s0 + r5 * s1 + r8 * s2);
      }
    }
    if (what == 2) f = inside ? mk3<double>(mx, my, mz) : mk3<double>(0, 0, 0);
    else {
      f = mk3<double>(hx, hy, hz);
      if (what == 0 && inside) { f.x += mx; f.y += my; f.z += mz; }
    }
  } else if (KIND == UK_ARC) {
    if (what != 2) f = arc_field(g.arc + (size_t)u.y * RADB200_ARC_STRIDE, q);
  } else {
    if (what != 2) {
      const double *b = g.bkg + 3 * (size_t)u.y;
      f = mk3<double>(__ldg(b), __ldg(b + 1), __ldg(b + 2));
    }
  }
  const double *F = Tr + 12;  // s*M
  return mk3<double>(__ldg(F + 0) * f.x + __ldg(F + 1) * f.y + __ldg(F + 2) * f.z,
                     __ldg(F + 3) * f.x + __ldg(F + 4) * f.y + __ldg(F + 5) * f.z,
                     __ldg(F + 6) * f.x + __ldg(F + 7) * f.y + __ldg(F + 8) * f.z);
}

// Units [ub, ue) of one kind; gridDim.y splits them into chunks.  With one
// chunk the result goes to out directly (accumulate: out += result), else to
// the chunk's slice of the partial buffer.
//
// Cuboids: bound by the FP64 pipe (about 430 operations a pair, 65-70% of its
// rate) and the latency between them.  4 CTAs per SM (128 registers): 3.94e9
// pairs in 136 ms, 2.9e10 pairs/s; 143 ms at 3 CTAs (158 registers); 490 ms
// with the term-by-term formula.
template <typename T, int KIND>
__global__ void __launch_bounds__(128, KIND == UK_REC ? 4 : 1) field_kernel(GeomView g, const double *__restrict__ pts, int64_t npts, int what,
                                                    double *__restrict__ out, int ub, int ue, int chunk, int accumulate)
{
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int u0 = ub + blockIdx.y * chunk, u1 = min(ue, u0 + chunk);
  bool active = i < npts;
  V3<double> P = mk3<double>(0, 0, 0);
  if (active) P = mk3<double>(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
  double ax = 0, ay = 0, az = 0;
  for (int u = u0; u < u1; u++) {
    int4 un = __ldg(g.units + u);
    V3<double> f = eval_unit<T, KIND>(g, un, P, what);
    ax += f.x; ay += f.y; az += f.z;
  }
  if (active) {
    double *o = out + ((size_t)blockIdx.y * npts + i) * 3;
    if (accumulate) { o[0] += ax; o[1] += ay; o[2] += az; }
    else { o[0] = ax; o[1] = ay; o[2] = az; }
  }
}

// out[i] (=|+=) sum_c partial[c][i], fixed order c = 0..nc-1
__global__ void chunk_reduce_kernel(const double *__restrict__ part, int nc, int64_t n3, double *__restrict__ out, int accumulate)
{
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  double s = accumulate ? out[i] : 0.0;
  for (int c = 0; c < nc; c++) s += part[(size_t)c * n3 + i];
  out[i] = s;
}

// All polyhedra are tetrahedra, FP64 vertex/edge form one by one (the mesh form
// serves B and H; this the rest).  A block of 128 threads takes 128 points and
// walks its unit range in tiles of 32 units whose records -- tetrahedron
// record, image transform, magnetization -- it first stages in shared memory.
constexpr int TET_TILE = 32;
constexpr int TET_U = TET_REC_FIELD + 21 + 3;  // record, Minv V sM (21), M (3)

__global__ void __launch_bounds__(128) field_tet_kernel(GeomView g, const double *__restrict__ pts, int64_t npts, int what,
                                                        double *__restrict__ out, int ub, int ue, int chunk, int accumulate)
{
  __shared__ double su[TET_TILE * TET_U];
  const int tid = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * 128 + tid;
  const int u0 = ub + blockIdx.y * chunk, u1 = min(ue, u0 + chunk);
  V3<double> P = mk3<double>(0, 0, 0);
  if (i < npts) P = mk3<double>(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
  double acc[3] = {0, 0, 0};
  for (int base = u0; base < u1; base += TET_TILE) {
    const int cnt = min(TET_TILE, u1 - base);
    __syncthreads();
    for (int e = tid; e < cnt * TET_U; e += 128) {
      const int k = e / TET_U, f = e - k * TET_U;
      const int4 un = __ldg(g.units + base + k);  // {kind, polyhedron, transform, ..}
      double v;
      if (f < TET_REC_FIELD) v = __ldg(g.tetrec + (size_t)__ldg(g.tetidx + un.y) * TET_REC_FIELD + f);
      else if (f < TET_REC_FIELD + 21) v = __ldg(g.trf + (size_t)un.z * RADB200_TRF_STRIDE + (f - TET_REC_FIELD));
      else v = __ldg(g.poly + (size_t)un.y * RADB200_POLY_STRIDE + 3 + (f - TET_REC_FIELD - 21));
      su[e] = v;
    }
    __syncthreads();
    for (int k = 0; k < cnt; k++) {
      const double *rec = su + k * TET_U, *Tr = rec + TET_REC_FIELD, *F = Tr + 12, *M = Tr + 21;
      const double dx = P.x - Tr[9], dy = P.y - Tr[10], dz = P.z - Tr[11];
      const V3<double> q = mk3<double>(Tr[0] * dx + Tr[1] * dy + Tr[2] * dz, Tr[3] * dx + Tr[4] * dy + Tr[5] * dz,
                                       Tr[6] * dx + Tr[7] * dy + Tr[8] * dz);
      double h[3];
      const int in = tet_fast<double, false, true>(rec, q, h);
      if (what == 2) h[0] = h[1] = h[2] = 0.0;
      if (what != 1 && in) { h[0] += M[0]; h[1] += M[1]; h[2] += M[2]; }
      acc[0] += F[0] * h[0] + F[1] * h[1] + F[2] * h[2];
      acc[1] += F[3] * h[0] + F[4] * h[1] + F[5] * h[2];
      acc[2] += F[6] * h[0] + F[7] * h[1] + F[8] * h[2];
    }
  }
  if (i < npts) {
    double *o = out + ((size_t)blockIdx.y * npts + i) * 3;
    if (accumulate) { o[0] += acc[0]; o[1] += acc[1]; o[2] += acc[2]; }
    else { o[0] = acc[0]; o[1] = acc[1]; o[2] = acc[2]; }
  }
}

// Triangle-face records (TRI_REC): a thread per polyhedron.
__global__ void tri_record_kernel(GeomView g, int n_poly, double *__restrict__ tri)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_poly) return;
  // the reference's polygon face form uses this 15-digit pi (radplnr2.cpp:32)
  const double CH = 1.0 / (4.0 * 3.14159265358979);
  const double *pr = g.poly + (size_t)p * RADB200_POLY_STRIDE;
  const int f0 = g.poly_info[4 * p], nf = g.poly_info[4 * p + 1];
  for (int f = f0; f < f0 + nf; f++) {
    const double *R = g.face + (size_t)f * RADB200_FACE_STRIDE;
    const double *vt = g.vtx2d + 2 * (size_t)g.face_vtx[2 * f];
    double *o = tri + (size_t)f * TRI_REC;
    const double n[3] = {R[6], R[7], R[8]}, c = CH * (n[0] * pr[3] + n[1] * pr[4] + n[2] * pr[5]);
    double a2 = 0.0, cx = 0.0, cy = 0.0;
    for (int k = 0; k < 3; k++) {
      const double x = vt[2 * k], y = vt[2 * k + 1];
      double e[EDGE_REC];
      edge_record(vt, 3, k, e);
      if (k == 1) a2 = e[3];
      cx += x;
      cy += y;
      o[9 + k] = e[2];
      for (int d = 0; d < 3; d++) {
        o[3 * k + d] = x * R[d] + y * R[3 + d] + R[9] * R[6 + d];
        o[18 + 3 * k + d] = c * (e[1] * R[d] - e[0] * R[3 + d]);  // outward: direction turned by -90 degrees
      }
    }
    for (int d = 0; d < 3; d++) {
      o[12 + d] = a2 * n[d];
      o[15 + d] = -c * n[d];
    }
    o[27] = fmax(abs_rand(g.g, R[9]), fmax(abs_rand(g.g, vt[0] - cx / 3), abs_rand(g.g, vt[1] - cy / 3)));
  }
}

int launch_tri_records(const GeomView &g, int n_poly, double *tri, cudaStream_t st)
{
  tri_record_kernel<<<(n_poly + 127) / 128, 128, 0, st>>>(g, n_poly, tri);
  return check_launch("tri_record_kernel");
}

// Face-by-face field of polyhedra with triangle faces.  The general kernel
// above reads a face through a chain of dependent loads (polyhedron, face,
// vertices) and waits on it: FP64 pipe 25% busy, 6e7 tetrahedron pairs in 8.4
// ms.  Here a block stages the records of up to TRI_TILE faces of up to 16
// units in shared memory: FP64 pipe 62% busy, 3.7 ms (1.6e10 pairs/s); the
// reference's polygon formula took 28 ms.  5 CTAs per SM: without the bound the
// rarely called poly_special would set the kernel's registers (158; 6% slower).
constexpr int TRI_UNITS = 16;
__global__ void __launch_bounds__(128, 5) field_tri_kernel(GeomView g, const double *__restrict__ pts, int64_t npts, int what,
                                                        double *__restrict__ out, int ub, int ue, int chunk, int accumulate)
{
  __shared__ double sf[TRI_TILE * TRI_REC];
  __shared__ double su[TRI_UNITS * 24];  // point map (12), field map (9), magnetization (3)
  __shared__ int s_face[TRI_UNITS], s_end[TRI_UNITS + 1], s_unit[TRI_UNITS], s_trf[TRI_UNITS], s_n;
  const int tid = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * 128 + tid;
  const int u0 = ub + blockIdx.y * chunk, u1 = min(ue, u0 + chunk);
  V3<double> P = mk3<double>(0, 0, 0);
  if (i < npts) P = mk3<double>(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
  double acc[3] = {0, 0, 0};
  for (int base = u0; base < u1;) {
    __syncthreads();  // the previous tile's readers are done
    if (tid < 32) {
      // the units that fit: a running sum of their faces
      int4 un = make_int4(0, 0, 0, 0);
      int nf = 0, f0 = 0;
      const bool has = tid < TRI_UNITS && base + tid < u1;
      if (has) {
        un = __ldg(g.units + base + tid);
        f0 = __ldg(g.poly_info + 4 * un.y);
        nf = __ldg(g.poly_info + 4 * un.y + 1);
      }
      int sum = nf;
#pragma unroll
      for (int o = 1; o < TRI_UNITS; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (tid >= o) sum += v;
      }
      const unsigned fit = __ballot_sync(0xffffffffu, has && sum <= TRI_TILE);
      if (has) {
        s_face[tid] = f0;
        s_end[tid + 1] = sum;
        s_unit[tid] = un.y;
        s_trf[tid] = un.z;
      }
      if (tid == 0) {
        s_end[0] = 0;
        s_n = __popc(fit);
      }
    }
    __syncthreads();
    const int nu = s_n;
    for (int k = 0; k < nu; k++) {
      const int e0 = s_end[k] * TRI_REC, ne = (s_end[k + 1] - s_end[k]) * TRI_REC;
      const double *src = g.tri + (size_t)s_face[k] * TRI_REC;
      for (int e = tid; e < ne; e += 128) sf[e0 + e] = __ldg(src + e);
    }
    for (int e = tid; e < nu * 24; e += 128) {
      const int k = e / 24, f = e - 24 * k;
      su[e] = f < 21 ? __ldg(g.trf + (size_t)s_trf[k] * RADB200_TRF_STRIDE + f)
                     : __ldg(g.poly + (size_t)s_unit[k] * RADB200_POLY_STRIDE + 3 + (f - 21));
    }
    __syncthreads();
    unsigned special = 0;  // units whose short form has no value at this point
    auto point = [&](const double *Tr) {
      const double dx = P.x - Tr[9], dy = P.y - Tr[10], dz = P.z - Tr[11];
      return mk3<double>(Tr[0] * dx + Tr[1] * dy + Tr[2] * dz, Tr[3] * dx + Tr[4] * dy + Tr[5] * dz,
                         Tr[6] * dx + Tr[7] * dy + Tr[8] * dz);
    };
    auto add = [&](const double *F, double hx, double hy, double hz) {
      acc[0] += F[0] * hx + F[1] * hy + F[2] * hz;
      acc[1] += F[3] * hx + F[4] * hy + F[5] * hz;
      acc[2] += F[6] * hx + F[7] * hy + F[8] * hz;
    };
    for (int k = 0; k < nu; k++) {
      const double *Tr = su + 24 * k, *M = Tr + 21;
      const V3<double> q = point(Tr);
      double h[3] = {0, 0, 0};
      int inside = 1;
      for (int f = s_end[k]; f < s_end[k + 1]; f++) inside &= tri_face(sf + f * TRI_REC, q, h);
      if (what == 2) h[0] = h[1] = h[2] = 0.0;
      if (not_finite(h[0])) {
        special |= 1u << k;
        continue;
      }
      if (what != 1 && inside) { h[0] += M[0]; h[1] += M[1]; h[2] += M[2]; }
      add(Tr + 12, h[0], h[1], h[2]);
    }
    for (; special; special &= special - 1) {
      const int k = __ffs(special) - 1;
      const double *Tr = su + 24 * k, *M = Tr + 21;
      PolygonTerms t = poly_special(g.face, g.face_vtx, g.vtx2d, s_face[k], s_end[k + 1] - s_end[k],
                                    mk3<double>(M[0], M[1], M[2]), point(Tr), g.g);
      if (what == 0 && t.in) { t.x += M[0]; t.y += M[1]; t.z += M[2]; }
      add(Tr + 12, t.x, t.y, t.z);
    }
    base += nu;
  }
  if (i < npts) {
    double *o = out + ((size_t)blockIdx.y * npts + i) * 3;
    if (accumulate) { o[0] += acc[0]; o[1] += acc[1]; o[2] += acc[2]; }
    else { o[0] = acc[0]; o[1] = acc[1]; o[2] = acc[2]; }
  }
}

template <typename T, int KIND>
static int launch_kind(const GeomView &g, const double *d_pts, int64_t npts, int what, double *d_out, int ub, int ue,
                       int accumulate, DBuf &scratch, cudaStream_t st)
{
  const int TPB = 128;
  int64_t nblk = (npts + TPB - 1) / TPB;
  int nu = ue - ub;
  // split the unit range when the points alone give fewer than ~8 CTAs per SM
  int nchunk = 1;
  const int64_t target = 148 * 8;
  if (nblk < target) nchunk = (int)((target + nblk - 1) / nblk);
  if (nchunk > nu) nchunk = nu;
  if (nchunk > 65535) nchunk = 65535;
  int chunk = (nu + nchunk - 1) / nchunk;
  nchunk = (nu + chunk - 1) / chunk;
  dim3 grid((unsigned)nblk, (unsigned)nchunk);
  double *dst = d_out;
  if (nchunk > 1) {
    RB_TRY(scratch.alloc((size_t)nchunk * npts * 3 * sizeof(double)));
    dst = scratch.as<double>();
  }
  const int acc = nchunk > 1 ? 0 : accumulate;
  if constexpr (KIND == UK_TET) field_tet_kernel<<<grid, TPB, 0, st>>>(g, d_pts, npts, what, dst, ub, ue, chunk, acc);
  else if constexpr (KIND == UK_TRI) field_tri_kernel<<<grid, TPB, 0, st>>>(g, d_pts, npts, what, dst, ub, ue, chunk, acc);
  else field_kernel<T, KIND><<<grid, TPB, 0, st>>>(g, d_pts, npts, what, dst, ub, ue, chunk, acc);
  RB_TRY(check_launch("field_kernel"));
  if (nchunk == 1) return 0;
  int64_t n3 = npts * 3;
  chunk_reduce_kernel<<<(unsigned)((n3 + 255) / 256), 256, 0, st>>>(scratch.as<double>(), nchunk, n3, d_out, accumulate);
  return check_launch("chunk_reduce_kernel");
}

// RADB200_MESH_FORM=0 evaluates all-tetrahedron models one tetrahedron at a
// time instead of by their unique edges and faces (A/B comparisons)
static bool mesh_form_enabled()
{
  static int on = -1;
  if (on < 0) {
    const char *e = getenv("RADB200_MESH_FORM");
    on = (e && atoi(e) == 0) ? 0 : 1;
  }
  return on == 1;
}

int launch_field(const GeomView &g, const double *d_pts, int64_t npts, int what, int precision, double *d_out,
                 DBuf &scratch, cudaStream_t st)
{
  if (npts <= 0) return 0;
  if ((npts + 127) / 128 > INT32_MAX) { set_error("too many points"); return RADB200_E_ARG; }
  if (g.n_units == 0) {
    RB_CUDA(cudaMemsetAsync(d_out, 0, (size_t)npts * 3 * sizeof(double), st));
    return 0;
  }
  // units are ordered by kind (cuboids, polyhedra, arcs, backgrounds): one launch per kind present
  int acc = 0;
  for (int kind = 0; kind < 4; kind++) {
    int ub = g.ustart[kind], ue = g.ustart[kind + 1];
    if (ue <= ub) continue;
    int rc;
    if (kind == 0)
      rc = launch_kind<double, UK_REC>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    // the mesh form in FP64 only: with FP32 terms its largest per-point B
    // error on the 20,000-tetrahedron model was 2.1e-6 against 7.6e-7 for the
    // tetrahedra one by one, at a 1.25x speed-up (1.42x in FP64)
    else if (kind == 1 && g.fast && g.all_tets && g.mesh.n_tiles > 0 && what != 2 && precision != 1 &&
             mesh_form_enabled())
      rc = launch_mesh_field(g, d_pts, npts, what, d_out, acc, scratch, st);
    else if (kind == 1 && g.fast && g.all_tets)
      rc = (precision == 1) ? launch_tet32_field(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st)
                            : launch_kind<double, UK_TET>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    else if (kind == 1 && g.fast)
      rc = (precision == 1) ? launch_kind<float, UK_POLY_FAST>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st)
                            : launch_kind<double, UK_POLY_FAST>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    else if (kind == 1 && g.tri)
      rc = launch_kind<double, UK_TRI>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    else if (kind == 1)
      rc = launch_kind<double, UK_POLY>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    else if (kind == 2)
      rc = launch_kind<double, UK_ARC>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    else
      rc = launch_kind<double, UK_BKG>(g, d_pts, npts, what, d_out, ub, ue, acc, scratch, st);
    RB_TRY(rc);
    acc = 1;
  }
  return 0;
}

__global__ void edge_record_kernel(const int *__restrict__ face_vtx, const double *__restrict__ vtx2d, int n_face,
                                   double *__restrict__ edge)
{
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_face) return;
  const int v0 = face_vtx[2 * f], nv = face_vtx[2 * f + 1];
  for (int j = 0; j < nv; j++) edge_record(vtx2d + 2 * (size_t)v0, nv, j, edge + EDGE_REC * ((size_t)v0 + j));
}

int launch_edge_records(const int *face_vtx, const double *vtx2d, int n_face, double *edge, cudaStream_t st)
{
  if (n_face <= 0) return 0;
  edge_record_kernel<<<(n_face + 127) / 128, 128, 0, st>>>(face_vtx, vtx2d, n_face, edge);
  return check_launch("edge_record_kernel");
}

// out_i = rowT_i * in_i  (3x3 per element)
__global__ void rowtrans_kernel(const double *__restrict__ rowT, const double *__restrict__ in, double *__restrict__ out, int n)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double *R = rowT + 9 * (size_t)i;
  double x = in[3 * i], y = in[3 * i + 1], z = in[3 * i + 2];
  out[3 * i] = R[0] * x + R[1] * y + R[2] * z;
  out[3 * i + 1] = R[3] * x + R[4] * y + R[5] * z;
  out[3 * i + 2] = R[6] * x + R[7] * y + R[8] * z;
}

int launch_rowtrans_vec(const double *rowT, const double *in, double *out, int n, cudaStream_t st)
{
  if (n <= 0) return 0;
  rowtrans_kernel<<<(n + 127) / 128, 128, 0, st>>>(rowT, in, out, n);
  return check_launch("rowtrans_kernel");
}

// ---------------------------------------------------------------------------
// Relativistic electron trajectories (FldPtcTrj).  The reference integrates
// x(y), x'(y), z(y), z'(y) with the field of the whole source evaluated at
// every Runge-Kutta stage (radTPrtclTrj::TrjEqs, cpp/src/core/radptrj.h:91-105;
// RungeKutta4 / Tabulation / RungeKuttaStep5 / AutoPropagate,
// radptrj.cpp:94-240).  The stages of one trajectory are a dependent chain,
// each a field evaluation over all sources, so a trajectory's time is that
// evaluation's latency.  A cluster of up to 8 CTAs carries one trajectory.  At
// every stage its warps take groups of 32 work items -- a (source, image) unit,
// or one node of an arc's trapezoid rule, whose nodes one after another were
// half of a stage -- one item per lane; each group's sum goes to every CTA's
// shared memory; after one cluster barrier every warp adds the groups up, in an
// order that does not depend on the cluster's size, and every thread advances
// an identical copy of the integrator state, so the control flow (the step-size
// control included) stays uniform.  Many trajectories take smaller clusters.
// 401 points through 300 cuboids with 4 images and a racetrack: 51 ms with one
// CTA each, 13.5 ms with 8.
// ---------------------------------------------------------------------------
constexpr int TRJ_THREADS = 256;
constexpr int TRJ_GROUPS = 512;  // groups of work items; larger models put several items on a lane

struct TrjArgs {
  double y0, step, ctm;  // start, tabulation step (mm), charge / momentum (1 / (T mm))
  int np, adaptive, max_steps;
  long long max_evals;   // field evaluations allowed per trajectory (bounds the kernel's run time)
  double prec[4], eps_tol;
  const int2 *items;     // {unit or -1, node of an arc or -1}
  int n_items, per_lane, n_groups;
};

// what a CTA carries through the evaluations
struct TrjCtx {
  double (*sum)[TRJ_GROUPS][3];  // [2]: the groups' sums, alternating
  int parity, rank, size;
};

__device__ __forceinline__ V3<double> trj_item(const GeomView &g, int2 it, V3<double> P)
{
  const int4 u = __ldg(g.units + it.x);
  if (u.x == 0) return eval_unit<double, UK_REC>(g, u, P, 0);
  if (u.x == 1) return eval_unit<double, UK_POLY>(g, u, P, 0);
  if (u.x == 3) return eval_unit<double, UK_BKG>(g, u, P, 0);
  const double *Tr = g.trf + (size_t)u.z * RADB200_TRF_STRIDE, *F = Tr + 12;
  const double dx = P.x - Tr[9], dy = P.y - Tr[10], dz = P.z - Tr[11];
  double f;
  V3<double> v = arc_node(g.arc + (size_t)u.y * RADB200_ARC_STRIDE,
                          mk3<double>(Tr[0] * dx + Tr[1] * dy + Tr[2] * dz, Tr[3] * dx + Tr[4] * dy + Tr[5] * dz,
                                      Tr[6] * dx + Tr[7] * dy + Tr[8] * dz),
                          it.y, f);
  v = mk3<double>(f * v.x, f * v.y, f * v.z);
  return mk3<double>(F[0] * v.x + F[1] * v.y + F[2] * v.z, F[3] * v.x + F[4] * v.y + F[5] * v.z,
                     F[6] * v.x + F[7] * v.y + F[8] * v.z);
}

__device__ __forceinline__ double warp_add(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// B at P from every item; every thread gets the sum
__device__ V3<double> trj_block_field(const GeomView &g, const TrjArgs &a, V3<double> P, TrjCtx &c)
{
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  c.parity ^= 1;
  double(*sum)[3] = c.sum[c.parity];
  for (int gr = c.rank * (TRJ_THREADS / 32) + warp; gr < a.n_groups; gr += c.size * (TRJ_THREADS / 32)) {
    double ax = 0, ay = 0, az = 0;
    for (int q = 0; q < a.per_lane; q++) {
      const int i = (gr * a.per_lane + q) * 32 + lane;
      if (i >= a.n_items) break;
      const int2 it = __ldg(a.items + i);
      if (it.x < 0) continue;
      const V3<double> f = trj_item(g, it, P);
      ax += f.x; ay += f.y; az += f.z;
    }
    __syncwarp();
    ax = warp_add(ax);
    ay = warp_add(ay);
    az = warp_add(az);
    if (lane < c.size) {
      double *dst = cl.map_shared_rank(&sum[gr][0], lane);
      dst[0] = ax;
      dst[1] = ay;
      dst[2] = az;
    }
  }
  // the other half of the buffer takes the next evaluation: a CTA that is
  // ahead by one cannot touch what a slower one still reads
  cl.sync();
  double bx = 0, by = 0, bz = 0;
  for (int gr = lane; gr < a.n_groups; gr += 32) {
    bx += sum[gr][0];
    by += sum[gr][1];
    bz += sum[gr][2];
  }
  return mk3<double>(warp_add(bx), warp_add(by), warp_add(bz));
}

// dF/dy for F = (x, x', z, z') at longitudinal position s
__device__ void trj_eqs(const GeomView &g, const TrjArgs &a, double s, const double *F, double *dF, TrjCtx &c,
                        long long &ne)
{
  ne++;
  double xd = F[1], zd = F[3];
  double xdxd = xd * xd, zdzd = zd * zd, xdzd = xd * zd;
  double buf = a.ctm * sqrt(1.0 + xdxd + zdzd);
  V3<double> B = trj_block_field(g, a, mk3<double>(F[0], s, F[2]), c);
  dF[0] = xd;
  dF[1] = -buf * (zd * B.y - (1.0 + xdxd) * B.z + xdzd * B.x);
  dF[2] = zd;
  dF[3] = buf * (xd * B.y - (1.0 + zdzd) * B.x + xdzd * B.z);
}

// classical fourth-order step of size h from (x, y) with slope dydx
__device__ void trj_rk4(const GeomView &g, const TrjArgs &a, const double *y, const double *dydx, double x, double h,
                        double *yout, TrjCtx &c, long long &ne)
{
  double hh = 0.5 * h, h6 = h / 6.0, xh = x + hh;
  double yt[4], dyt[4], dym[4];
  for (int i = 0; i < 4; i++) yt[i] = y[i] + hh * dydx[i];
  trj_eqs(g, a, xh, yt, dyt, c, ne);
  for (int i = 0; i < 4; i++) yt[i] = y[i] + hh * dyt[i];
  trj_eqs(g, a, xh, yt, dym, c, ne);
  for (int i = 0; i < 4; i++) {
    yt[i] = y[i] + h * dym[i];
    dym[i] += dyt[i];
  }
  trj_eqs(g, a, x + h, yt, dyt, c, ne);
  for (int i = 0; i < 4; i++) yout[i] = y[i] + h6 * (dydx[i] + dyt[i] + 2.0 * dym[i]);
}

// step-doubling control: one step of size h against two of h/2, accepted when
// the difference over prec, over eps_tol, is at most 1; 0 ok, 1 step too small,
// 2 evaluation budget spent, 3 no acceptable step within the shrink limit
__device__ int trj_step5(const GeomView &g, const TrjArgs &a, double *y, double *dydx, double *x, double htry,
                         double *hdid, double *hnext, TrjCtx &c, long long &ne)
{
  const double PGROW = -0.2, PSHRNK = -0.25, FCOR = 1.0 / 15.0, SAFETY = 0.9, ERRCON = 6.0e-04;
  double xsav = *x, h = htry, ysav[4], dysav[4], ytemp[4];
  for (int i = 0; i < 4; i++) { ysav[i] = y[i]; dysav[i] = dydx[i]; }
  for (int it = 0; it < 200; it++) {
    if (ne > a.max_evals) return 2;
    double hh = 0.5 * h;
    trj_rk4(g, a, ysav, dysav, xsav, hh, ytemp, c, ne);
    *x = xsav + hh;
    trj_eqs(g, a, *x, ytemp, dydx, c, ne);
    trj_rk4(g, a, ytemp, dydx, *x, hh, y, c, ne);
    *x = xsav + h;
    if (*x == xsav) return 1;
    trj_rk4(g, a, ysav, dysav, xsav, h, ytemp, c, ne);
    double errmax = 0.0;
    for (int i = 0; i < 4; i++) {
      ytemp[i] = y[i] - ytemp[i];
      double t = fabs(ytemp[i] / a.prec[i]);
      if (errmax < t) errmax = t;
    }
    errmax /= a.eps_tol;
    if (errmax <= 1.0) {
      *hdid = h;
      *hnext = (errmax > ERRCON ? SAFETY * h * exp(PGROW * log(errmax)) : 4.0 * h);
      for (int i = 0; i < 4; i++) y[i] += ytemp[i] * FCOR;
      return 0;
    }
    if (!(errmax < 1e300)) return 3;  // non-finite error: no step will be accepted
    h *= SAFETY * exp(PSHRNK * log(errmax));
  }
  return 3;
}

// adaptive propagation of y from x1 to x2; 0 ok, 1 step too small, 2 step limit, 3 failure
__device__ int trj_propagate(const GeomView &g, const TrjArgs &a, double *ystart, double x1, double x2, double h1,
                             double hmin, TrjCtx &c, long long &ne)
{
  double x = x1, h = (x2 > x1) ? fabs(h1) : -fabs(h1), y[4], dydx[4], hdid, hnext;
  for (int i = 0; i < 4; i++) y[i] = ystart[i];
  for (int n = 1; n <= a.max_steps; n++) {
    trj_eqs(g, a, x, y, dydx, c, ne);
    if ((x + h - x2) * (x + h - x1) > 0.0) h = x2 - x;
    int rc = trj_step5(g, a, y, dydx, &x, h, &hdid, &hnext, c, ne);
    if (rc) return rc;
    if ((x - x2) * (x2 - x1) >= 0.0) {
      for (int i = 0; i < 4; i++) ystart[i] = y[i];
      return 0;
    }
    if (fabs(hnext) <= hmin) return 1;
    h = hnext;
  }
  return 2;
}

// out[(b * np + i) * 5 + (y, x, x', z, z')]; status[b]: 0 ok, else the failure code
__global__ void __launch_bounds__(TRJ_THREADS) trajectory_kernel(GeomView g, TrjArgs a, const double *__restrict__ init,
                                                                double *__restrict__ out, int *__restrict__ status)
{
  __shared__ double sums[2][TRJ_GROUPS][3];
  TrjCtx c;
  c.sum = sums;
  c.parity = 0;
  c.rank = (int)cooperative_groups::this_cluster().block_rank();
  c.size = (int)cooperative_groups::this_cluster().num_blocks();
  const int b = blockIdx.x / c.size;
  const bool writer = c.rank == 0 && threadIdx.x == 0;
  double Y[4], dY[4];
  for (int k = 0; k < 4; k++) Y[k] = init[4 * b + k];
  double x = a.y0, hmin = 1e-10 * a.step;
  int rc = 0;
  long long ne = 0;
  // every CTA of the cluster has started before any writes to another's sums
  cooperative_groups::this_cluster().sync();
  for (int i = 0; i < a.np; i++) {
    if (!a.adaptive) trj_eqs(g, a, x, Y, dY, c, ne);
    if (writer) {
      double *o = out + ((size_t)b * a.np + i) * 5;
      o[0] = x;
      for (int k = 0; k < 4; k++) o[1 + k] = Y[k];
    }
    if (i == a.np - 1 || rc) break;
    double x1 = x + a.step;
    if (a.adaptive) rc = trj_propagate(g, a, Y, x, x1, a.step, hmin, c, ne);
    else trj_rk4(g, a, Y, dY, x, a.step, Y, c, ne);
    x = x1;
    if (rc) {
      // rows after a failed interval repeat the last good state's position with NaN
      for (int j = i + 1; j < a.np && writer; j++) {
        double *o = out + ((size_t)b * a.np + j) * 5;
        for (int k = 0; k < 5; k++) o[k] = __longlong_as_double(0x7ff8000000000000LL);
      }
      break;
    }
  }
  if (writer) status[b] = rc;
  cooperative_groups::this_cluster().sync();  // no CTA leaves while another may still write to its sums
}

int launch_trajectories(const GeomView &g, double energy_gev, const double *d_init, int n_traj, double y0, double y1,
                        int np, const double *prec, const int2 *d_items, int n_items, double *d_out, int *d_status,
                        cudaStream_t st)
{
  if (n_traj <= 0) return 0;
  TrjArgs a;
  a.y0 = y0;
  a.np = np;
  a.step = (np > 1) ? (y1 - y0) / (double)(np - 1) : 0.0;
  a.ctm = -2.99792458e+05 / (1.e+09 * energy_gev);  // electron charge over momentum
  a.adaptive = prec != nullptr;
  a.max_steps = 5000;
  a.max_evals = 40LL * np + 40000;
  a.eps_tol = 1.0;
  for (int k = 0; k < 4; k++) a.prec[k] = prec ? (prec[k] == 0.0 ? 1e23 : prec[k]) : 1.0;
  a.items = d_items;
  a.n_items = n_items;
  a.per_lane = std::max(1, (n_items + 32 * TRJ_GROUPS - 1) / (32 * TRJ_GROUPS));
  a.n_groups = (n_items + 32 * a.per_lane - 1) / (32 * a.per_lane);
  // CTAs per trajectory: as many as leave every CTA an SM of its own and
  // every warp a group
  int size = 8;
  while (size > 1 && ((int64_t)n_traj * size > 148 || (size / 2) * (TRJ_THREADS / 32) >= a.n_groups)) size /= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_traj * size);
  cfg.blockDim = dim3(TRJ_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  RB_CUDA(cudaLaunchKernelEx(&cfg, trajectory_kernel, g, a, d_init, d_out, d_status));
  return check_launch("trajectory_kernel");
}

}  // namespace rb
