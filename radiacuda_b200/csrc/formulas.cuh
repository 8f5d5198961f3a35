// formulas.cuh -- device formulas of the Radia field sources (sm_100a).
//
// Closed forms, restated for the device from the reference CPU code (the GPU
// port of the reference differs in places; the CPU code is the contract):
//   cuboid tensor / current field    radTRecMag::B_comp      radrec.cpp:49-315
//   polygon face integrals           radTPolygon::B_comp     radplnr2.cpp:29-388
//   arc current (trapezoid in phi)   radTArcCur::B_compWithTrapeth radarccu.cpp:30-236
// All functions are templated on the arithmetic type T (double, or float for
// the single-precision field option); guards follow radTConvergRepair
// (radcnvrg.h:85-91) with the magnitudes passed in Guard.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "elem64.cuh"

namespace rb {

template <typename T> struct V3 { T x, y, z; };
template <typename T> __host__ __device__ __forceinline__ V3<T> mk3(T x, T y, T z) { V3<T> r; r.x = x; r.y = y; r.z = z; return r; }

struct Guard { double absr, relr, zeror; };

template <typename T> __device__ __forceinline__ T fabsT(T x) { return x < T(0) ? -x : x; }
__device__ __forceinline__ double logT(double x) { return log(x); }
__device__ __forceinline__ float logT(float x) { return logf(x); }
__device__ __forceinline__ double atan2T(double y, double x) { return atan2(y, x); }
__device__ __forceinline__ float atan2T(float y, float x) { return atan2f(y, x); }
__device__ __forceinline__ double sqrtT(double x) { return sqrt(x); }
__device__ __forceinline__ float sqrtT(float x) { return sqrtf(x); }

// radTConvergRepair::AbsRandMagnitude (radcnvrg.h:85-91)
template <typename T> __device__ __forceinline__ T abs_rand(const Guard &g, T A)
{
  if (g.absr == 0.0 && g.relr == 0.0 && g.zeror == 0.0) return T(0);
  T fromrel = T(g.relr) * A;
  T amax = (fromrel < T(g.absr)) ? T(g.absr) : fromrel;
  return (A != T(0)) ? amax : ((amax < T(g.zeror)) ? T(g.zeror) : amax);
}

// ---- cuboid -------------------------------------------------------------------
// Q of a uniformly magnetized cuboid (radrec.cpp:115-283) at q from its centre:
//   4 pi Tx = sum of 8 arctan(+-y_j z_k / (x_i D_ijk)),
//   4 pi Sz = -log of a product of 8 factors (z_k + D_ijk)^+-1,  and cyclic.
// Evaluated term by term as the reference does, a pair costs 24 quotients
// inside the arctangents, 18 in their addition formulas, 12 in the logarithms,
// and 6 arctangents: about 2,000 FP64 issue slots.  Here:
//   - each arctangent is the argument of x D + i (+-y z); the arguments of a
//     face add up in the product of its four numbers, both faces of an axis in
//     one more product, so an axis costs no quotients and one arctangent.  The
//     product knows its angle modulo 2 pi.  The turns come from the quadrants
//     of the two face products: seen from the point a face has a solid angle
//     in (0, pi), or in (0, 2 pi) when the point projects into it (then all
//     four arguments are positive and the product's quadrant cannot be
//     mistaken by rounding).  Quadrant centres are within pi/4 of the angles,
//     two faces and their product within 3 pi/4 of a multiple of 2 pi;
//   - z + D with z < 0 cancels; there it is rho^2 / (|z| + D), rho^2 =
//     x^2 + y^2.  For z_0 and z_1 of one sign the rho^2 cancel between the two
//     ends and only the logarithm's sign changes; otherwise they stay as a
//     factor.  No quotient, no cancellation, one logarithm of a ratio per axis.
//   - the third diagonal entry is what the trace leaves: 0 outside, -1 inside.
// elem64.cuh has the square root, arctangent and logarithm.

// The product of one face's four numbers: offset a along the axis, p_jk the
// products of the other two offsets, u = p00 p01, v = p10 p11, D_jk the
// distances of its corners
RB_HD void cuboid_face(double a, double p00, double p01, double p10, double p11, double u, double v, double D00, double D01,
                       double D10, double D11, double &re, double &im)
{
  const double r0 = a * D00, r1 = a * D01, r2 = a * D10, r3 = a * D11;
  const double e0 = fma(r0, r1, u), f0 = fma(p00, r1, -(r0 * p01));
  const double e1 = fma(r2, r3, v), f1 = fma(r2, p11, -(p10 * r3));
  re = fma(e0, e1, -(f0 * f1));
  im = fma(e0, f1, f0 * e1);
}
// The face's angle by quadrant, in units of pi/4 (the centre), with the sign of
// its offset a, which the product carries; inner: the point projects into it
RB_HD int cuboid_face_quadrant(double a, double re, double im, bool inner)
{
  const int s = hi32(a);
  const int c = hi32(re) < 0 ? ((hi32(im) ^ s) < 0 ? 5 : 3) : ((hi32(im) ^ s) < 0 ? (inner ? 7 : -1) : 1);
  return s < 0 ? -c : c;
}
RB_HD int plain_quadrant(double re, double im)
{
  return hi32(re) < 0 ? (hi32(im) < 0 ? -3 : 3) : (hi32(im) < 0 ? -1 : 1);
}

// one axis: T of the faces at a0 and a1
RB_HD double cuboid_axis_T(double a0, double a1, double p00, double p01, double p10, double p11, double D000,
                           double D001, double D010, double D011, double D100, double D101, double D110, double D111,
                           bool inner)
{
  const double u = p00 * p01, v = p10 * p11;
  double re0, im0, re1, im1;
  cuboid_face(a0, p00, p01, p10, p11, u, v, D000, D001, D010, D011, re0, im0);
  cuboid_face(a1, p00, p01, p10, p11, u, v, D100, D101, D110, D111, re1, im1);
  const double re = fma(re0, re1, im0 * im1), im = fma(im0, re1, -(re0 * im1));
  const int c0 = cuboid_face_quadrant(a0, re0, im0, inner), c1 = cuboid_face_quadrant(a1, re1, im1, inner);
  return angle64(im, re, (c0 - c1 - plain_quadrant(re, im) + 4) >> 3);
}

// one axis: the logarithm of S.  b_ijk = |a_k| + D of the corners, the axis's
// own index last; n2, d2 the rho^2 products that replace the cancelling sums
// when the two offsets have opposite signs (mixed); neg: the first one is negative
RB_HD double cuboid_axis_L(double b000, double b001, double b010, double b011, double b100, double b101, double b110,
                           double b111, double n2, double d2, bool mixed, bool neg)
{
  const double e = b001 * b111, f = b101 * b011, g = b100 * b010, h = b000 * b110;
  const double n = mixed ? (e * h) * n2 : e * g, d = mixed ? (f * g) * d2 : f * h;
  const double L = log_ratio64(n, d);
  return neg && !mixed ? -L : L;
}

// Replacement near a corner with the length guards on (radrec.cpp:131-156):
// z + D below 10 times the guard of D becomes rho^2 / (2 |z|).  b = |z| + D.
__device__ __forceinline__ double cuboid_guard_b(const Guard &g, double z, double D, double rho2)
{
  const double b = fabs(z) + D, R = 10.0 * abs_rand(g, D);
  if (z < 0.0) return rho2 < R * b ? 2.0 * fabs(z) : b;
  return b < R ? 0.5 * rho2 / fabs(z) : b;
}

// q = observation point RELATIVE TO THE CUBOID CENTRE (object frame), hd =
// half dimensions.  Returns 1 if strictly inside.  Writes the symmetric tensor
// entries T = (Txx,Tyy,Tzz) and S = (Sx,Sy,Sz) times 4 pi (the caller scales
// by CUBOID_C):
//   Q = [[Tx,-Sz,-Sy],[-Sz,Ty,-Sx],[-Sy,-Sx,Tz]]    (radrec.cpp:265-283)
constexpr double CUBOID_C = 1.0 / (4.0 * 3.141592653589793238);
__device__ __forceinline__ int cuboid_TS(V3<double> q, V3<double> hd, const Guard &g, V3<double> &Tt, V3<double> &Ss)
{
  // the signs of the widths, if negative, turn the sign of the whole tensor
  const int ws = hi32(hd.x) ^ hi32(hd.y) ^ hi32(hd.z);
  const double hx = fabs(hd.x), hy = fabs(hd.y), hz = fabs(hd.z);
  double x0 = -q.x - hx, x1 = -q.x + hx;
  double y0 = -q.y - hy, y1 = -q.y + hy;
  double z0 = -q.z - hz, z1 = -q.z + hz;
  // on a face plane the guards step off it; without guards the normal entry
  // of the tensor is undefined there (0/0 in the reference), NaN
  int nan = 0;
  if (x0 == 0.0 || x1 == 0.0) {
    const double r = abs_rand(g, hx);
    if (x0 == 0.0) x0 = r;
    if (x1 == 0.0) x1 = r;
    nan |= (r == 0.0);
  }
  if (y0 == 0.0 || y1 == 0.0) {
    const double r = abs_rand(g, hy);
    if (y0 == 0.0) y0 = r;
    if (y1 == 0.0) y1 = r;
    nan |= (r == 0.0) << 1;
  }
  if (z0 == 0.0 || z1 == 0.0) {
    const double r = abs_rand(g, hz);
    if (z0 == 0.0) z0 = r;
    if (z1 == 0.0) z1 = r;
    nan |= (r == 0.0) << 2;
  }
  // Q has no dimension: bring extreme units (products of 16 lengths occur) to
  // around 1 by a power of two
  {
    const int top = max(max(hi32(fabs(x0)), max(hi32(fabs(x1)), hi32(fabs(y0)))),
                        max(hi32(fabs(y1)), max(hi32(fabs(z0)), hi32(fabs(z1)))));
    const int e = (top >> 20) - 1023;
    if (e > 40 || e < -40) {
      const double sc = scalbn(1.0, e > 1000 ? -1000 : -e);
      x0 *= sc; x1 *= sc; y0 *= sc; y1 *= sc; z0 *= sc; z1 *= sc;
    }
  }
  const bool mx = (hi32(x0) & ~hi32(x1)) < 0, my = (hi32(y0) & ~hi32(y1)) < 0, mz = (hi32(z0) & ~hi32(z1)) < 0;
  const double xx0 = x0 * x0, xx1 = x1 * x1, yy0 = y0 * y0, yy1 = y1 * y1, zz0 = z0 * z0, zz1 = z1 * z1;
  const double xy00 = xx0 + yy0, xy01 = xx0 + yy1, xy10 = xx1 + yy0, xy11 = xx1 + yy1;
  const double D000 = sqrt64(xy00 + zz0), D001 = sqrt64(xy00 + zz1), D010 = sqrt64(xy01 + zz0), D011 = sqrt64(xy01 + zz1);
  const double D100 = sqrt64(xy10 + zz0), D101 = sqrt64(xy10 + zz1), D110 = sqrt64(xy11 + zz0), D111 = sqrt64(xy11 + zz1);
  Tt.x = cuboid_axis_T(x0, x1, y0 * z0, y0 * z1, y1 * z0, y1 * z1, D000, D001, D010, D011, D100, D101, D110, D111, my && mz);
  Tt.y = cuboid_axis_T(y0, y1, x0 * z0, x0 * z1, x1 * z0, x1 * z1, D000, D001, D100, D101, D010, D011, D110, D111, mx && mz);
  const bool in = mx && my && mz;
  Tt.z = (in ? -4.0 * 3.141592653589793238 : 0.0) - (Tt.x + Tt.y);
  const double xz00 = xx0 + zz0, xz01 = xx0 + zz1, xz10 = xx1 + zz0, xz11 = xx1 + zz1;
  const double yz00 = yy0 + zz0, yz01 = yy0 + zz1, yz10 = yy1 + zz0, yz11 = yy1 + zz1;
  const double ax0 = fabs(x0), ax1 = fabs(x1), ay0 = fabs(y0), ay1 = fabs(y1), az0 = fabs(z0), az1 = fabs(z1);
  if (g.absr > 0.0 && fmin(fmin(fmin(D000, D001), fmin(D010, D011)), fmin(fmin(D100, D101), fmin(D110, D111))) < 10.0 * g.absr) {
    Ss.z = cuboid_axis_L(cuboid_guard_b(g, z0, D000, xy00), cuboid_guard_b(g, z1, D001, xy00), cuboid_guard_b(g, z0, D010, xy01),
                         cuboid_guard_b(g, z1, D011, xy01), cuboid_guard_b(g, z0, D100, xy10), cuboid_guard_b(g, z1, D101, xy10),
                         cuboid_guard_b(g, z0, D110, xy11), cuboid_guard_b(g, z1, D111, xy11), xy10 * xy01, xy00 * xy11, mz, hi32(z0) < 0);
    Ss.y = cuboid_axis_L(cuboid_guard_b(g, y0, D000, xz00), cuboid_guard_b(g, y1, D010, xz00), cuboid_guard_b(g, y0, D001, xz01),
                         cuboid_guard_b(g, y1, D011, xz01), cuboid_guard_b(g, y0, D100, xz10), cuboid_guard_b(g, y1, D110, xz10),
                         cuboid_guard_b(g, y0, D101, xz11), cuboid_guard_b(g, y1, D111, xz11), xz10 * xz01, xz00 * xz11, my, hi32(y0) < 0);
    Ss.x = cuboid_axis_L(cuboid_guard_b(g, x0, D000, yz00), cuboid_guard_b(g, x1, D100, yz00), cuboid_guard_b(g, x0, D001, yz01),
                         cuboid_guard_b(g, x1, D101, yz01), cuboid_guard_b(g, x0, D010, yz10), cuboid_guard_b(g, x1, D110, yz10),
                         cuboid_guard_b(g, x0, D011, yz11), cuboid_guard_b(g, x1, D111, yz11), yz10 * yz01, yz00 * yz11, mx, hi32(x0) < 0);
  } else {
    Ss.z = cuboid_axis_L(az0 + D000, az1 + D001, az0 + D010, az1 + D011, az0 + D100, az1 + D101, az0 + D110, az1 + D111,
                         xy10 * xy01, xy00 * xy11, mz, hi32(z0) < 0);
    Ss.y = cuboid_axis_L(ay0 + D000, ay1 + D010, ay0 + D001, ay1 + D011, ay0 + D100, ay1 + D110, ay0 + D101, ay1 + D111,
                         xz10 * xz01, xz00 * xz11, my, hi32(y0) < 0);
    Ss.x = cuboid_axis_L(ax0 + D000, ax1 + D100, ax0 + D001, ax1 + D101, ax0 + D010, ax1 + D110, ax0 + D011, ax1 + D111,
                         yz10 * yz01, yz00 * yz11, mx, hi32(x0) < 0);
  }
  // S is minus the logarithm
  Ss = mk3<double>(flip_sign(Ss.x, ~ws), flip_sign(Ss.y, ~ws), flip_sign(Ss.z, ~ws));
  Tt = mk3<double>(flip_sign(Tt.x, ws), flip_sign(Tt.y, ws), flip_sign(Tt.z, ws));
  if (nan) {
    const double bad = __longlong_as_double(0x7ff8000000000000LL);
    if (nan & 1) Tt.x = bad;
    if (nan & 2) Tt.y = bad;
    if (nan & 4) Tt.z = bad;
  }
  return in;
}

// x0 T0 + x1 T1 of one axis: the faces' own angles, weighted by their offsets
RB_HD double cuboid_axis_xT(double a0, double a1, double p00, double p01, double p10, double p11, double D000, double D001,
                            double D010, double D011, double D100, double D101, double D110, double D111, bool inner)
{
  const double u = p00 * p01, v = p10 * p11;
  double re, im;
  cuboid_face(a0, p00, p01, p10, p11, u, v, D000, D001, D010, D011, re, im);
  const double t0 = angle64(im, re, (cuboid_face_quadrant(a0, re, im, inner) - plain_quadrant(re, im) + 4) >> 3);
  cuboid_face(a1, p00, p01, p10, p11, u, v, D100, D101, D110, D111, re, im);
  const double t1 = angle64(im, re, (cuboid_face_quadrant(a1, re, im, inner) - plain_quadrant(re, im) + 4) >> 3);
  return fma(a0, t0, -(a1 * t1));
}
// log((z0 + D0) / (z1 + D1)) along an edge at rho^2 from the point's axis, from
// b = |z| + D (a sum with z < 0 is rho^2 / b)
RB_HD double cuboid_edge_L(double b0, double b1, double rho2, bool mixed, bool neg)
{
  return log_ratio64(mixed ? rho2 : (neg ? b1 : b0), mixed ? b0 * b1 : (neg ? b0 : b1));
}

// Field of a current-carrying cuboid (radrec.cpp:183-249, J branch), q
// relative to the centre, J in A/mm^2; returns B (= H) in T.  Single blocks
// of coils lie on the critical path of a trajectory's field evaluations: with
// the elements of cuboid_TS, 12 logarithms and 6 arctangents without quotients.
__device__ __forceinline__ V3<double> cuboid_J(V3<double> q, V3<double> hd, V3<double> J, const Guard &g)
{
  // the signs of the widths, if negative, turn the field (cuboid_TS)
  const int ws = hi32(hd.x) ^ hi32(hd.y) ^ hi32(hd.z);
  const double hx = fabs(hd.x), hy = fabs(hd.y), hz = fabs(hd.z);
  double x0 = -q.x - hx, x1 = -q.x + hx, y0 = -q.y - hy, y1 = -q.y + hy, z0 = -q.z - hz, z1 = -q.z + hz;
  int nan = 0;
  if (x0 == 0. || x1 == 0.) { const double r = abs_rand(g, hx); if (x0 == 0.) x0 = r; if (x1 == 0.) x1 = r; nan |= r == 0.; }
  if (y0 == 0. || y1 == 0.) { const double r = abs_rand(g, hy); if (y0 == 0.) y0 = r; if (y1 == 0.) y1 = r; nan |= (r == 0.) << 1; }
  if (z0 == 0. || z1 == 0.) { const double r = abs_rand(g, hz); if (z0 == 0.) z0 = r; if (z1 == 0.) z1 = r; nan |= (r == 0.) << 2; }
  const bool mx = (hi32(x0) & ~hi32(x1)) < 0, my = (hi32(y0) & ~hi32(y1)) < 0, mz = (hi32(z0) & ~hi32(z1)) < 0;
  const bool nx = hi32(x0) < 0, ny = hi32(y0) < 0, nz = hi32(z0) < 0;
  const double xx0 = x0 * x0, xx1 = x1 * x1, yy0 = y0 * y0, yy1 = y1 * y1, zz0 = z0 * z0, zz1 = z1 * z1;
  const double D000 = sqrt64(xx0 + yy0 + zz0), D001 = sqrt64(xx0 + yy0 + zz1), D010 = sqrt64(xx0 + yy1 + zz0),
               D011 = sqrt64(xx0 + yy1 + zz1), D100 = sqrt64(xx1 + yy0 + zz0), D101 = sqrt64(xx1 + yy0 + zz1),
               D110 = sqrt64(xx1 + yy1 + zz0), D111 = sqrt64(xx1 + yy1 + zz1);
  const double xT = cuboid_axis_xT(x0, x1, y0 * z0, y0 * z1, y1 * z0, y1 * z1, D000, D001, D010, D011, D100, D101, D110, D111, my && mz);
  const double yT = cuboid_axis_xT(y0, y1, x0 * z0, x0 * z1, x1 * z0, x1 * z1, D000, D001, D100, D101, D010, D011, D110, D111, mx && mz);
  const double zT = cuboid_axis_xT(z0, z1, x0 * y0, x0 * y1, x1 * y0, x1 * y1, D000, D010, D100, D110, D001, D011, D101, D111, mx && my);
  const bool near = g.absr > 0.0 && fmin(fmin(fmin(D000, D001), fmin(D010, D011)), fmin(fmin(D100, D101), fmin(D110, D111))) < 10.0 * g.absr;
  auto b = [&](double z, double D, double rho2) { return near ? cuboid_guard_b(g, z, D, rho2) : fabs(z) + D; };
  auto L = [&](double c0, double c1, double D0, double D1, double rho2, bool m, bool n) {
    return cuboid_edge_L(b(c0, D0, rho2), b(c1, D1, rho2), rho2, m, n);
  };
  const double lz00 = L(z0, z1, D000, D001, xx0 + yy0, mz, nz), lz01 = L(z0, z1, D010, D011, xx0 + yy1, mz, nz),
               lz10 = L(z0, z1, D100, D101, xx1 + yy0, mz, nz), lz11 = L(z0, z1, D110, D111, xx1 + yy1, mz, nz);
  const double ly00 = L(y0, y1, D000, D010, xx0 + zz0, my, ny), ly01 = L(y0, y1, D001, D011, xx0 + zz1, my, ny),
               ly10 = L(y0, y1, D100, D110, xx1 + zz0, my, ny), ly11 = L(y0, y1, D101, D111, xx1 + zz1, my, ny);
  const double lx00 = L(x0, x1, D000, D100, yy0 + zz0, mx, nx), lx01 = L(x0, x1, D001, D101, yy0 + zz1, mx, nx),
               lx10 = L(x0, x1, D010, D110, yy1 + zz0, mx, nx), lx11 = L(x0, x1, D011, D111, yy1 + zz1, mx, nx);
  V3<double> bv = mk3<double>(xT + y0 * (lz10 - lz00) + y1 * (lz01 - lz11) + z0 * (ly10 - ly00) + z1 * (ly01 - ly11),
                              yT + x0 * (lz01 - lz00) + x1 * (lz10 - lz11) + z0 * (lx10 - lx00) + z1 * (lx01 - lx11),
                              zT + y0 * (lx01 - lx00) + y1 * (lx10 - lx11) + x0 * (ly01 - ly00) + x1 * (ly10 - ly11));
  if (nan) {  // on a face plane without guards the angle is undefined, as in the reference
    const double bad = __longlong_as_double(0x7ff8000000000000LL);
    if (nan & 1) bv.x = bad;
    if (nan & 2) bv.y = bad;
    if (nan & 4) bv.z = bad;
  }
  const double c = flip_sign(0.0001, ws);
  return mk3<double>(c * (J.y * bv.z - J.z * bv.y), c * (J.z * bv.x - J.x * bv.z), c * (J.x * bv.y - J.y * bv.x));
}

// Planar polygon face integrals (Sx,Sy,Sz) at a point given in the face frame
// (px,py,pz), vertices (counter-clockwise) in shared or global memory.
// Returns 1 when the point is on the inner side of the face plane (z > 0).
// radTPolygon::B_comp, radplnr2.cpp:29-388 (B/H/PreRelax paths), term by term.
// Used where blocks of the interaction matrix must follow the reference's own
// rounding: close to slivers its terms lose 1e-12 of a block and more, which
// chi = 1000 amplifies, and relaxed magnetizations are compared at 1e-9.
// Fields use polygon_S below (2,500 against about 170 issue slots a face).
template <typename T, typename VP>
__device__ __forceinline__ int polygon_S_terms(const VP *vtx, int nv, T coordz, T cx, T cy, V3<T> P,
                                          const Guard &g, T &Sx_o, T &Sy_o, T &Sz_o)
{
  const T Max_k = T(1.E+09);
  T arx = abs_rand(g, T(vtx[0]) - cx), ary = abs_rand(g, T(vtx[1]) - cy);
  T arz = abs_rand(g, coordz);
  if (arz < arx) arz = arx;
  if (arz < ary) arz = ary;
  T relr = abs_rand(g, T(1));
  T z = coordz - P.z;
  if (z == T(0)) z = arz;
  T ze2 = z * z;
  T f2x = T(vtx[0]) - P.x, f2y = T(vtx[1]) - P.y;
  T addx = -P.x, addy = -P.y;
  T x1 = f2x, y1 = f2y;
  if (x1 == T(0)) { x1 = arx; f2x += arx; addx += arx; }
  if (y1 == T(0)) { y1 = ary; f2y += ary; addy += ary; }
  T x1e2 = x1 * x1;
  T Sx = 0, Sy = 0, sum_atan = 0, arg_logs2 = 1;
  const T MaxRel = T(1.E-07);
  const T tiny = sizeof(T) == 8 ? T(1e-50) : T(1e-30);
  for (int i = 0; i < nv; i++) {
    T x2, y2;
    if (i != nv - 1) { x2 = T(vtx[2 * (i + 1)]) + addx; y2 = T(vtx[2 * (i + 1) + 1]) + addy; }
    else { x2 = f2x; y2 = f2y; }
    if (x2 == T(0)) { x2 = arx; f2x += arx; addx += arx; }
    if (y2 == T(0)) { y2 = ary; f2y += ary; addy += ary; }
    T x2e2 = x2 * x2;
    T x2mx1 = x2 - x1, y2my1 = y2 - y1;
    if (fabsT(x2mx1) * Max_k > fabsT(y2my1)) {
      T k = y2my1 / x2mx1;
      T b = y1 - k * x1;
      if (b == T(0)) {
        b = ary; y1 += ary; y2my1 -= ary; k = y2my1 / x2mx1;
        f2y += ary; addy += ary;
      }
      T bk = b * k, ke2 = k * k, be2 = b * b, twob = T(2) * b;
      T ke2p1 = ke2 + T(1);
      if (ke2p1 == T(0)) ke2p1 = relr;
      T sqrtke2p1 = sqrtT(ke2p1);
      T kx1 = k * x1, kx2 = k * x2;
      T bpkx1 = y1, bpkx2 = y2;
      T bpkx1e2 = bpkx1 * bpkx1, bpkx2e2 = bpkx2 * bpkx2;
      T kx1mb = -b + kx1, kx2mb = -b + kx2;
      T R1 = sqrtT(x1e2 + bpkx1e2 + ze2), R2 = sqrtT(x2e2 + bpkx2e2 + ze2);
      T x1e2pze2 = x1e2 + ze2, x2e2pze2 = x2e2 + ze2;
      T bkpx1pke2x1 = bk + ke2p1 * x1, bkpx2pke2x2 = bk + ke2p1 * x2;
      T kze2 = k * ze2, ke2ze2 = k * kze2;
      T ke2ze2mbe2 = ke2ze2 - be2, ke2ze2pbe2 = ke2ze2 + be2;
      T bx1 = b * x1, bx2 = b * x2;
      T R1pbpkx1 = bpkx1 + R1, R2pbpkx2 = bpkx2 + R2;
      T arR2 = T(100) * abs_rand(g, R2), arR1 = T(100) * abs_rand(g, R1);
      T mR1 = MaxRel * R1, mR2 = MaxRel * R2;
      if (arR1 > mR1) arR1 = mR1;
      if (arR2 > mR2) arR2 = mR2;
      if ((R1pbpkx1 < arR1) && (R1 > T(100) * arR1) && ((x1e2 + ze2) < bpkx1e2 * MaxRel))
        R1pbpkx1 = T(0.5) * (x1e2 + ze2) / fabsT(bpkx1);
      if ((R2pbpkx2 < arR2) && (R2 > T(100) * arR2) && ((x2e2 + ze2) < bpkx2e2 * MaxRel))
        R2pbpkx2 = T(0.5) * (x2e2 + ze2) / fabsT(bpkx2);
      T A1 = -(ke2ze2pbe2 * (bx1 + kze2) * R1pbpkx1 + kze2 * twob * x1e2pze2);
      T A2 = (ke2ze2pbe2 * kx1mb * R1pbpkx1 + ke2ze2mbe2 * x1e2pze2) * z;
      T A3 = ke2ze2pbe2 * (bx2 + kze2) * R2pbpkx2 + kze2 * twob * x2e2pze2;
      T A4 = (ke2ze2pbe2 * kx2mb * R2pbpkx2 + ke2ze2mbe2 * x2e2pze2) * z;
      sum_atan += atan2T(A1 * A4 + A3 * A2, A2 * A4 - A1 * A3);
      T L1 = bkpx1pke2x1 / sqrtke2p1 + R1, L2 = bkpx2pke2x2 / sqrtke2p1 + R2;
      T be2pze2 = be2 + ze2;
      if ((L1 < arR1) && (R1 > T(100) * arR1) && ((be2pze2 + T(2) * bk * x1) < x1e2 * ke2p1 * MaxRel))
        L1 = T(0.5) * be2pze2 / (fabsT(x1) * sqrtke2p1);
      if ((L2 < arR2) && (R2 > T(100) * arR2) && ((be2pze2 + T(2) * bk * x2) < x2e2 * ke2p1 * MaxRel))
        L2 = T(0.5) * be2pze2 / (fabsT(x2) * sqrtke2p1);
      if (L1 == T(0)) L1 = tiny;
      if (L2 == T(0)) L2 = tiny;
      T sl1 = logT(L2 / L1) / sqrtke2p1;
      if (R1pbpkx1 == T(0)) R1pbpkx1 = tiny;
      arg_logs2 *= (R2pbpkx2 / R1pbpkx1);
      Sx += -k * sl1;
      Sy += sl1;
    }
    x1 = x2; y1 = y2; x1e2 = x2e2;
  }
  if (arg_logs2 <= T(0)) arg_logs2 = tiny;
  Sx += logT(arg_logs2);
  Sx_o = Sx; Sy_o = Sy; Sz_o = sum_atan;
  return z > T(0);
}

// ---- polygon face ---------------------------------------------------------------
// Face integrals (Sx, Sy, Sz) of a planar polygon at a point given in the face
// frame (radTPolygon::B_comp, radplnr2.cpp:29-388; B/H/PreRelax paths):
//   (Sx, Sy) = sum over edges of (-ty, tx) L,   Sz = solid angle, > 0 below,
// with (tx, ty) the edge's direction and L = edge_log64.  The reference writes
// each edge as y = k x + b: its log(L2/L1)/sqrt(k^2+1) is this L, the
// remaining product of its logarithm telescopes to the vertical edges' share,
// and its arctangents of one edge each sum to the solid angle of the polygon.
// Here an edge costs one logarithm and no quotient (directions and lengths
// are kept per vertex, EdgeRec), neighbouring edges share a distance, and a
// triangle of the fan takes one arctangent (Van Oosterom-Strackee), its
// numerator z times twice its area: a triangle face about 170 FP64 operations
// against 2,500 issue slots.
constexpr int EDGE_REC = 4;
// of polygon vertex j: direction (2) and length of the edge to the next
// vertex, twice the area of the fan triangle (0, j, j + 1).  An edge between
// two equal vertices (a collapsed face) has direction zero and adds nothing.
RB_HD void edge_record(const double *vtx, int nv, int j, double *e)
{
  const int k = j + 1 < nv ? j + 1 : 0;
  const double ex = vtx[2 * k] - vtx[2 * j], ey = vtx[2 * k + 1] - vtx[2 * j + 1];
  const double l = sqrt(ex * ex + ey * ey);
  const double fx = vtx[2 * j] - vtx[0], fy = vtx[2 * j + 1] - vtx[1];
  e[0] = l > 0.0 ? ex / l : 0.0;
  e[1] = l > 0.0 ? ey / l : 0.0;
  e[2] = l;
  e[3] = fx * ey - fy * ex;
}

// half the solid angle of a triangle whose plane is at height z: a2 twice its
// area, offsets (x, y, z) and distances of its vertices
__device__ __forceinline__ double half_solid_angle(double z, double zz, double a2, double x0, double y0, double R0,
                                                   double x1, double y1, double R1, double x2, double y2, double R2)
{
  const double d01 = fma(x0, x1, fma(y0, y1, zz)), d02 = fma(x0, x2, fma(y0, y2, zz)), d12 = fma(x1, x2, fma(y1, y2, zz));
  return atan2_64(z * a2, fma(fma(R0, R1, d01), R2, fma(d02, R1, d12 * R0)));
}

// polygon_S_terms as a call, for the points where the short form has no value
// or not the reference's: S (3) and the inner-side flag
struct PolygonTerms {
  double x, y, z;
  int in;
};
__device__ __noinline__ static PolygonTerms polygon_special(const double *vtx, int nv, double coordz, V3<double> P, Guard g)
{
  double cx = 0, cy = 0;
  for (int k = 0; k < nv; k++) { cx += vtx[2 * k]; cy += vtx[2 * k + 1]; }
  PolygonTerms t;
  t.in = polygon_S_terms<double, double>(vtx, nv, coordz, cx / nv, cy / nv, P, g, t.x, t.y, t.z);
  return t;
}
// D of an edge's ends (edge_D64), NaN for a point within twice the guard's step
// of the edge or an end (without guards, on it): there the integrals are what
// the reference's own steps leave of infinite ones
__device__ __noinline__ static double edge_D64_off(double ax, double ay, double az, double Ra, double bx, double by, double bz,
                                                   double Rb, double l, double step)
{
  const double cx = ay * bz - az * by, cy = az * bx - ax * bz, cz = ax * by - ay * bx, r = 2.0 * step;
  if (fmin(Ra, Rb) <= r || cx * cx + cy * cy + cz * cz <= (r * l) * (r * l)) return __longlong_as_double(0x7ff8000000000000LL);
  return edge_D64(ax, ay, az, Ra, bx, by, bz, Rb);
}
RB_HD bool not_finite(double x) { return (hi32(x) & 0x7ff00000) == 0x7ff00000; }

// vtx: nv counter-clockwise vertices in the face frame; er: their edge records
// (null: formed here).  A point with z == 0 steps off the plane by the length
// guard; without guards it is on the outer side (-0: the solid angle's limit
// from there, which the flag and the M path agree with).  Boundary points, and
// distances whose squares overflow, take the reference's terms.
__device__ __forceinline__ int polygon_S(const double *vtx, const double *er, int nv, double coordz, V3<double> P,
                                         const Guard &g, double &Sx, double &Sy, double &Sz)
{
  double z = coordz - P.z;
  double step = 0.0;
  if (z == 0.0) {
    double cx = 0, cy = 0;
    for (int k = 0; k < nv; k++) { cx += vtx[2 * k]; cy += vtx[2 * k + 1]; }
    step = fmax(abs_rand(g, coordz), fmax(abs_rand(g, vtx[0] - cx / nv), abs_rand(g, vtx[1] - cy / nv)));
    z = step > 0.0 ? step : -0.0;
  }
  const double zz = z * z;
  auto edge = [&](int j, double *e) {
    if (er) {
      const double2 a = __ldg(reinterpret_cast<const double2 *>(er + EDGE_REC * j)),
                    b = __ldg(reinterpret_cast<const double2 *>(er + EDGE_REC * j) + 1);
      e[0] = a.x; e[1] = a.y; e[2] = b.x; e[3] = b.y;
    } else edge_record(vtx, nv, j, e);
  };
  auto edge_L = [&](double ax, double ay, double Ra, double bx, double by, double Rb, double l) {
    const double S = Ra + Rb;
    double L;
    edge_logs64<1>(&S, &l, &L, [&](int) { return edge_D64_off(ax, ay, z, Ra, bx, by, z, Rb, l, step); });
    return L;
  };
  auto finish = [&]() -> int {
    if (!not_finite(Sx)) return z > 0.0;
    const PolygonTerms t = polygon_special(vtx, nv, coordz, P, g);
    Sx = t.x; Sy = t.y; Sz = t.z;
    return t.in;
  };
  const double x0 = vtx[0] - P.x, y0 = vtx[1] - P.y, R0 = sqrt64(fma(x0, x0, fma(y0, y0, zz)));
  double e[EDGE_REC];
  if (nv == 3) {
    const double x1 = vtx[2] - P.x, y1 = vtx[3] - P.y, R1 = sqrt64(fma(x1, x1, fma(y1, y1, zz)));
    const double x2 = vtx[4] - P.x, y2 = vtx[5] - P.y, R2 = sqrt64(fma(x2, x2, fma(y2, y2, zz)));
    edge(0, e);
    double L = edge_L(x0, y0, R0, x1, y1, R1, e[2]);
    Sx = -e[1] * L;
    Sy = e[0] * L;
    edge(2, e);
    L = edge_L(x2, y2, R2, x0, y0, R0, e[2]);
    Sx = fma(-e[1], L, Sx);
    Sy = fma(e[0], L, Sy);
    edge(1, e);
    L = edge_L(x1, y1, R1, x2, y2, R2, e[2]);
    Sx = fma(-e[1], L, Sx);
    Sy = fma(e[0], L, Sy);
    Sz = 2.0 * half_solid_angle(z, zz, e[3], x0, y0, R0, x1, y1, R1, x2, y2, R2);
    return finish();
  }
  double xp = x0, yp = y0, Rp = R0;
  Sx = Sy = Sz = 0.0;
  for (int j = 0; j < nv; j++) {
    double xn = x0, yn = y0, Rn = R0;
    if (j + 1 < nv) {
      xn = vtx[2 * j + 2] - P.x;
      yn = vtx[2 * j + 3] - P.y;
      Rn = sqrt64(fma(xn, xn, fma(yn, yn, zz)));
    }
    edge(j, e);
    const double L = edge_L(xp, yp, Rp, xn, yn, Rn, e[2]);
    Sx = fma(-e[1], L, Sx);
    Sy = fma(e[0], L, Sy);
    if (j > 0 && j + 1 < nv) Sz += 2.0 * half_solid_angle(z, zz, e[3], x0, y0, R0, xp, yp, Rp, xn, yn, Rn);
    xp = xn; yp = yn; Rp = Rn;
  }
  return finish();
}

// ---- triangle face in three dimensions -------------------------------------------
// For polyhedra of triangles (meshes): the same face integral from the face's
// own vertices in the object frame.  Record, TRI_REC doubles:
//   [0,9) vertices  [9,12) edge lengths (01 12 20)  [12,15) m, normal times
//   twice the area  [15,18) -c n  [18,27) c nu of the edges (outward, in plane)
//   [27] the length guard's step off the plane (0 without guards)
// c = M.n / (4 pi) with the face form's pi, so that H += sum L c nu - half angle * 2 c n.
constexpr int TRI_REC = 28;

// adds the face's H to h; returns 1 when q is on the inner side (polygon_S).
// h[0] is not finite after a face at whose boundary points, or at whose
// distance, only the reference's terms have a value: poly_special then.
__device__ __forceinline__ int tri_face(const double *rec, V3<double> q, double *h)
{
  double x[3], y[3], z[3], R[3], S[3], L[3];
#pragma unroll
  for (int k = 0; k < 3; k++) { x[k] = rec[3 * k] - q.x; y[k] = rec[3 * k + 1] - q.y; z[k] = rec[3 * k + 2] - q.z; }
  const double m0 = rec[12], m1 = rec[13], m2 = rec[14];
  double num = fma(x[0], m0, fma(y[0], m1, z[0] * m2));
  if (num == 0.0 && !(rec[27] > 0.0)) num = -0.0;
  else if (num == 0.0) {  // on the plane, guards on
    const double mm = sqrt64(fma(m0, m0, fma(m1, m1, m2 * m2))), s = rec[27] / mm;
    for (int k = 0; k < 3; k++) { x[k] += s * m0; y[k] += s * m1; z[k] += s * m2; }
    num = rec[27] * mm;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) R[k] = sqrt64(fma(x[k], x[k], fma(y[k], y[k], z[k] * z[k])));
  S[0] = R[0] + R[1]; S[1] = R[1] + R[2]; S[2] = R[2] + R[0];
  edge_logs64<3>(S, rec + 9, L, [&](int e) {
    const int b = e == 2 ? 0 : e + 1;
    return edge_D64_off(x[e], y[e], z[e], R[e], x[b], y[b], z[b], R[b], rec[9 + e], rec[27]);
  });
  const double d01 = fma(x[0], x[1], fma(y[0], y[1], z[0] * z[1])), d12 = fma(x[1], x[2], fma(y[1], y[2], z[1] * z[2])),
               d02 = fma(x[0], x[2], fma(y[0], y[2], z[0] * z[2]));
  const double w = 2.0 * atan2_64(num, fma(fma(R[0], R[1], d01), R[2], fma(d02, R[1], d12 * R[0])));
#pragma unroll
  for (int c = 0; c < 3; c++)
    h[c] += fma(L[0], rec[18 + c], fma(L[1], rec[21 + c], fma(L[2], rec[24 + c], w * rec[15 + c])));
  return num > 0.0;
}

// H of a polyhedron by the reference's terms, faces [f0, f0 + nf); in: 1 when q
// is on the inner side of all
__device__ __noinline__ static PolygonTerms poly_special(const double *face, const int *face_vtx, const double *vtx2d, int f0,
                                                         int nf, V3<double> M, V3<double> q, Guard g)
{
  // the reference's polygon face form uses this 15-digit pi (radplnr2.cpp:32)
  const double CH = 1.0 / (4.0 * 3.14159265358979);
  PolygonTerms h{0.0, 0.0, 0.0, 1};
  for (int f = f0; f < f0 + nf; f++) {
    const double *R = face + (size_t)f * RADB200_FACE_STRIDE;
    const V3<double> pl = mk3<double>(R[0] * q.x + R[1] * q.y + R[2] * q.z, R[3] * q.x + R[4] * q.y + R[5] * q.z,
                                      R[6] * q.x + R[7] * q.y + R[8] * q.z);
    const PolygonTerms s = polygon_special(vtx2d + 2 * (size_t)face_vtx[2 * f], face_vtx[2 * f + 1], R[9], pl, g);
    const double w = -CH * (R[6] * M.x + R[7] * M.y + R[8] * M.z);
    h.x += w * (R[0] * s.x + R[3] * s.y + R[6] * s.z);
    h.y += w * (R[1] * s.x + R[4] * s.y + R[7] * s.z);
    h.z += w * (R[2] * s.x + R[5] * s.y + R[8] * s.z);
    h.in &= s.in;
  }
  return h;
}

// u + D of two legs of D, other legs' squares q; direct when D was raised to the
// reference's least value (then q / (|u| + D) is another number)
__device__ __forceinline__ double arc_sum(double u, double D, double q, bool raised)
{
  return u < 0.0 && !raised ? q / (fabs(u) + D) : u + D;
}
// The logarithms that take D11 and D21 (arc_node) within 1e-5 of the arc's lower
// inner or outer corner edge, where the reference raises these to 1e-5
__device__ __noinline__ static double2 arc_corner_logs(double r1, double r2, double z1, double z2, double h1, double h2, double zz1,
                                                       double D11, double D12, double D21, double D22, double least)
{
  const bool c1 = h1 + z1 * z1 < least, c2 = h2 + z1 * z1 < least;
  return make_double2(log(arc_sum(r1, D11, zz1, c1) / arc_sum(r2, D21, zz1, c2)),
                      log(arc_sum(z1, D11, h1, c1) / arc_sum(z2, D12, h1, false)) -
                          log(arc_sum(z1, D21, h2, c2) / arc_sum(z2, D22, h2, false)));
}

// Arc current field at q (object frame), record a = [cx cy cz rmin rmax
// phimin phimax h j nseg]; trapezoid rule in phi with nseg sectors
// (radTArcCur::B_compWithTrapeth, radarccu.cpp:30-236).
// One node i of the rule with its weight; the field is f times the nodes' sum.
// The reference's terms with the elements of the cuboid: a sum u + D that
// cancels for u < 0 is the square of the other legs over |u| + D, a pair of
// arctangents is the argument of one product, and the angle between the point
// and the node comes from their directions.
__device__ __forceinline__ V3<double> arc_node(const double *a, V3<double> P, int i, double &f)
{
  const double ZeroTol = 1.E-10, SP = 1.E-10;
  const double px = P.x - a[0], py = P.y - a[1], pz = P.z - a[2];
  const double Rmin = a[3], Rmax = a[4], Phimin = a[5], Phimax = a[6], Height = a[7], Jaz = a[8];
  const int nsec = (int)a[9];
  const double rr = px * px + py * py + SP, r = sqrt64(rr);
  // direction of the point, with SP on the y side as in the reference's arccosine of px / r
  const double ir = rcp64(r), cp = px * ir, spa = sqrt64(fma(py, py, SP)) * ir, sp = py < 0 ? -spa : spa;
  const double z1 = -Height / 2. - pz, z2 = z1 + Height;
  const double step = (Phimax - Phimin + SP) / nsec;
  double sph, cph;
  sincos(Phimin + SP + i * step, &sph, &cph);
  const double sdp = sph * cp - cph * sp, cdp = cph * cp + sph * sp;
  const double rs = r * fabs(sdp), rCos = r * cdp, r1 = Rmin - rCos, r2 = Rmax - rCos;
  const double z1z1 = z1 * z1, z2z2 = z2 * z2, ss = rs * rs, zz1 = z1z1 + ss, zz2 = z2z2 + ss;
  const double h1 = fma(r1, r1, ss), h2 = fma(r2, r2, ss);  // squared distances in the plane
  const double D11 = sqrt64(fmax(h1 + z1z1, ZeroTol)), D12 = sqrt64(fmax(h1 + z2z2, 1e-290));
  const double D21 = sqrt64(fmax(h2 + z1z1, ZeroTol)), D22 = sqrt64(fmax(h2 + z2z2, 1e-290));
  const double b1 = fabs(r1), b2 = fabs(r2), c1 = fabs(z1), c2 = fabs(z2);
  const bool mr = r1 < 0.0 && r2 > 0.0, nr = r1 < 0.0, mz = z1 < 0.0 && z2 > 0.0, nz = z1 < 0.0;
  double ln1 = cuboid_edge_L(b1 + D11, b2 + D21, zz1, mr, nr);         // log((r1 + D11) / (r2 + D21))
  const double ln2 = -cuboid_edge_L(b1 + D12, b2 + D22, zz2, mr, nr);  // log((r2 + D22) / (r1 + D12))
  double lz = cuboid_edge_L(c1 + D11, c2 + D12, h1, mz, nz) - cuboid_edge_L(c1 + D21, c2 + D22, h2, mz, nz);
  if (fmin(h1, h2) + z1z1 < ZeroTol) {
    const double2 t = arc_corner_logs(r1, r2, z1, z2, h1, h2, zz1, D11, D12, D21, D22, ZeroTol);
    ln1 = t.x;
    lz = t.y;
  }
  // arctan(z2 |r1| / (rs D12)) - arctan(z1 |r1| / (rs D11)), and the outer radius with the sign turned
  const double e1 = rs * D12, g1 = z2 * b1, e2 = rs * D11, g2 = z1 * b1;
  const double at1 = angle64(fma(g1, e2, -(e1 * g2)), fma(e1, e2, g1 * g2), 0);
  const double e3 = rs * D21, g3 = z1 * b2, e4 = rs * D22, g4 = z2 * b2;
  const double at2 = angle64(fma(g3, e4, -(e3 * g4)), fma(e3, e4, g3 * g4), 0);
  const double Buf = rs * ((r1 < 0 ? -at1 : at1) + (r2 < 0 ? -at2 : at2)) + z1 * ln1 + z2 * ln2;
  const double FBxy = D11 - D21 + D22 - D12 + rCos * (ln1 + ln2);
  const double FBz = Buf - rCos * lz;
  const double wgt = (i == 0 || i == nsec) ? 0.5 : 1.0;
  f = 0.0001 * Jaz * step;
  return mk3<double>(wgt * cph * FBxy, wgt * sph * FBxy, wgt * FBz);
}
__device__ __forceinline__ V3<double> arc_field(const double *a, V3<double> P)
{
  const int n = (int)a[9] + 1;
  V3<double> s = mk3<double>(0, 0, 0);
  double f = 0.0;
  for (int i = 0; i < n; i++) {
    const V3<double> v = arc_node(a, P, i, f);
    s.x += v.x; s.y += v.y; s.z += v.z;
  }
  return mk3<double>(f * s.x, f * s.y, f * s.z);
}

// ---------------------------------------------------------------------------
// Polyhedron, vertex/edge form.
//
// The field of a uniformly magnetized polyhedron is that of the surface
// charge sigma_f = M.n_f on its faces:
//   H(q) = 1/(4 pi) sum_f sigma_f I_f,   I_f = int_f (q - r')/|q - r'|^3 dS'
// and for a planar face   I_f = Omega_f n_f + sum_{e in f} nu_{e,f} L_e
// with Omega_f the signed solid angle of the face seen from q (sign of
// n_f.(q - face)), nu_{e,f} the outward in-plane normal of edge e in face f
// and L_e = int_e dl/|q - r'| = log1p(l (Ra + Rb + l) / D),
// D = Ra Rb + ra.rb  (evaluated as |ra x rb|^2 / (Ra Rb - ra.rb) when ra.rb < 0
// to avoid cancellation).  Solid angles per triangle by the Van Oosterom-
// Strackee formula, with the triple product taken from the face's fixed edge
// cross product (ra . m_t, m_t = (vb - va) x (vc - va)) so it does not cancel
// for distant points.  Per tetrahedron this is 4 sqrt, 6 log1p, 4 atan2,
// against 12 edge terms (24 sqrt, 24 log, 12 atan2) of the face-by-face form
// radplnr2.cpp:29-388; both are exact, so they agree to rounding away from
// the edges themselves.
//
// Topology record per polyhedron (built on the host from the face frames):
//   tinfo  = {v0, nv, e0, ne},  tinfo2 = {t0, nt, f0, nf}
//   tv[v]  vertex (object frame)          te[e] = {a, b} (local), tel[e] = l
//   tt[t]  = {a, b, c, f} (local), ttm[t] = m_t
//   tfn[f] = n_f
// Field mode adds per face a_f = sigma_f n_f and per edge g_e = sum_f sigma_f nu_{e,f};
// tensor mode uses per edge G_e = sum_f nu_{e,f} n_f^T (9 doubles).
struct TopoView {
  const int4 *tinfo, *tinfo2;
  const double *tv;     // [V*3]
  const int2 *te;       // [E]
  const double *tel;    // [E]
  const double *teg;    // [E*3] field coefficients g_e (or null)
  const double *teG;    // [E*9] tensor coefficients G_e (or null)
  const int4 *tt;       // [T]
  const double *ttm;    // [T*3]
  const double *tfn;    // [F*3]
  const double *tfa;    // [F*3] field coefficients a_f (or null)
};

constexpr int POLY_NV_FAST = 8;  // vertices handled in registers

// the vertex/edge forms' elements in either precision: distance, edge
// integral L (ends a, b, their distances and dot product d) and angle
__device__ __forceinline__ double edge_R(double x, double y, double z) { return sqrt64(fma(x, x, fma(y, y, z * z))); }
__device__ __forceinline__ float edge_R(float x, float y, float z) { return sqrtf(x * x + y * y + z * z); }
__device__ __forceinline__ double edge_L(double ax, double ay, double az, double Ra, double bx, double by, double bz,
                                         double Rb, double, double l)
{
  const double S = Ra + Rb;
  double L;
  edge_logs64<1>(&S, &l, &L, [&](int) { return edge_D64(ax, ay, az, Ra, bx, by, bz, Rb); });
  return L;
}
__device__ __forceinline__ float edge_L(float ax, float ay, float az, float Ra, float bx, float by, float bz, float Rb,
                                        float d, float l)
{
  float D;
  if (d >= 0.f) D = Ra * Rb + d;
  else {
    const float cx = ay * bz - az * by, cy = az * bx - ax * bz, cz = ax * by - ay * bx;
    D = (cx * cx + cy * cy + cz * cz) / (Ra * Rb - d);
  }
  return log1pf(l * (Ra + Rb + l) / D);
}
__device__ __forceinline__ double face_angle(double y, double x) { return atan2_64(y, x); }
__device__ __forceinline__ float face_angle(float y, float x) { return atan2f(y, x); }

// Solid angles and edge logs of polyhedron p at q (object frame).
// Accumulates H (field mode, a_f / g_e set) or the tensor Q (tensor mode).
// Returns 1 when q is inside.  T = arithmetic type after the FP64 vertex shift.
template <typename T, bool TENSOR>
__device__ __forceinline__ int poly_fast(const TopoView &tp, int p, V3<double> q, double *out)
{
  const double C = 1.0 / (4.0 * 3.141592653589793238);
  int4 i1 = __ldg(tp.tinfo + p), i2 = __ldg(tp.tinfo2 + p);
  const int v0 = i1.x, nv = i1.y, e0 = i1.z, ne = i1.w, t0 = i2.x, nt = i2.y, f0 = i2.z, nf = i2.w;
  T rx[POLY_NV_FAST], ry[POLY_NV_FAST], rz[POLY_NV_FAST], R[POLY_NV_FAST];
#pragma unroll
  for (int k = 0; k < POLY_NV_FAST; k++) {
    if (k < nv) {
      const double *v = tp.tv + 3 * (size_t)(v0 + k);
      rx[k] = T(__ldg(v) - q.x); ry[k] = T(__ldg(v + 1) - q.y); rz[k] = T(__ldg(v + 2) - q.z);
      R[k] = edge_R(rx[k], ry[k], rz[k]);
    } else {
      rx[k] = ry[k] = rz[k] = R[k] = T(0);
    }
  }
  double acc[9];
#pragma unroll
  for (int k = 0; k < 9; k++) acc[k] = 0.0;
  // edges
  for (int e = e0; e < e0 + ne; e++) {
    int2 ab = __ldg(tp.te + e);
    T l = T(__ldg(tp.tel + e));
    T ax = T(0), ay = T(0), az = T(0), Ra = T(0), bx = T(0), by = T(0), bz = T(0), Rb = T(0);
#pragma unroll
    for (int k = 0; k < POLY_NV_FAST; k++) {
      if (k == ab.x) { ax = rx[k]; ay = ry[k]; az = rz[k]; Ra = R[k]; }
      if (k == ab.y) { bx = rx[k]; by = ry[k]; bz = rz[k]; Rb = R[k]; }
    }
    T L = edge_L(ax, ay, az, Ra, bx, by, bz, Rb, ax * bx + ay * by + az * bz, l);
    double Ld = (double)L;
    if (TENSOR) {
      const double *G = tp.teG + 9 * (size_t)e;
#pragma unroll
      for (int k = 0; k < 9; k++) acc[k] += Ld * __ldg(G + k);
    } else {
      const double *g = tp.teg + 3 * (size_t)e;
      acc[0] += Ld * __ldg(g); acc[1] += Ld * __ldg(g + 1); acc[2] += Ld * __ldg(g + 2);
    }
  }
  // triangles -> face solid angles
  double omega_tot = 0.0;
  int fcur = -1;
  double om = 0.0;
  for (int t = t0; t <= t0 + nt; t++) {
    int4 tr = (t < t0 + nt) ? __ldg(tp.tt + t) : make_int4(0, 0, 0, -1);
    if (tr.w != fcur) {
      if (fcur >= 0) {  // flush face fcur
        const double *n = tp.tfn + 3 * (size_t)(f0 + fcur);
        if (TENSOR) {
          double n0 = __ldg(n), n1 = __ldg(n + 1), n2 = __ldg(n + 2);
          acc[0] += om * n0 * n0; acc[1] += om * n0 * n1; acc[2] += om * n0 * n2;
          acc[3] += om * n1 * n0; acc[4] += om * n1 * n1; acc[5] += om * n1 * n2;
          acc[6] += om * n2 * n0; acc[7] += om * n2 * n1; acc[8] += om * n2 * n2;
        } else {
          const double *a = tp.tfa + 3 * (size_t)(f0 + fcur);
          acc[0] += om * __ldg(a); acc[1] += om * __ldg(a + 1); acc[2] += om * __ldg(a + 2);
        }
        omega_tot += om;
      }
      fcur = tr.w;
      om = 0.0;
      if (t == t0 + nt) break;
    }
    T xa = 0, ya = 0, za = 0, Ra = 0, xb = 0, yb = 0, zb = 0, Rb = 0, xc = 0, yc = 0, zc = 0, Rc = 0;
#pragma unroll
    for (int k = 0; k < POLY_NV_FAST; k++) {
      if (k == tr.x) { xa = rx[k]; ya = ry[k]; za = rz[k]; Ra = R[k]; }
      if (k == tr.y) { xb = rx[k]; yb = ry[k]; zb = rz[k]; Rb = R[k]; }
      if (k == tr.z) { xc = rx[k]; yc = ry[k]; zc = rz[k]; Rc = R[k]; }
    }
    const double *m = tp.ttm + 3 * (size_t)t;
    T num = xa * T(__ldg(m)) + ya * T(__ldg(m + 1)) + za * T(__ldg(m + 2));
    T den = Ra * Rb * Rc + (xa * xb + ya * yb + za * zb) * Rc + (xa * xc + ya * yc + za * zc) * Rb +
            (xb * xc + yb * yc + zb * zc) * Ra;
    om += 2.0 * (double)face_angle(-num, den);
  }
#pragma unroll
  for (int k = 0; k < (TENSOR ? 9 : 3); k++) out[k] = C * acc[k];
  return omega_tot < -6.283185307179586;
}

// ---------------------------------------------------------------------------
// Tetrahedron, vertex/edge form with a fixed topology: edges (01 02 03 12 13
// 23), faces opposite each vertex, the face cross products m_t oriented
// outward on the host.  No index selection in the inner loop, everything
// unrolled.  Record (object frame), TET_REC_FIELD doubles:
//   [0,12) vertices  [12,18) edge lengths  [18,30) m_t  [30,42) a_f = sigma_f n_f
//   [42,60) g_e = sum_f sigma_f nu_{e,f}
// TET_REC_TENSOR doubles: [0,30) as above, [30,42) n_f, [42,78) the symmetric
// parts of G_e (xx xy xz yy yz zz each): the tensor is symmetric, so the
// antisymmetric parts cancel in its sum over edges.
constexpr int TET_REC_FIELD = 60, TET_REC_TENSOR = 78;
__host__ __device__ constexpr int tet_edge_a(int e) { return e < 3 ? 0 : (e < 5 ? 1 : 2); }
__host__ __device__ constexpr int tet_edge_b(int e) { return e == 0 ? 1 : e == 1 ? 2 : e == 2 ? 3 : e == 3 ? 2 : 3; }
// face f (opposite vertex f) = triangle (a, b, c)
__host__ __device__ constexpr int tet_face_a(int f) { return f == 0 ? 1 : 0; }
__host__ __device__ constexpr int tet_face_b(int f) { return f == 0 ? 2 : (f == 1 ? 2 : 1); }
__host__ __device__ constexpr int tet_face_c(int f) { return f == 3 ? 2 : 3; }
// index of the vertex pair (i < j) in the edge list
__host__ __device__ constexpr int tet_pair(int i, int j) { return i == 0 ? j - 1 : (i == 1 ? j + 1 : 5); }

template <bool SMEM>
__device__ __forceinline__ double rd_rec(const double *p)
{
  if (SMEM) return *p;
  return __ldg(p);
}

// SMEM: the record lives in shared memory (plain loads instead of __ldg).
template <typename T, bool TENSOR, bool SMEM = false>
__device__ __forceinline__ int tet_fast(const double *__restrict__ rec, V3<double> q, double *out)
{
  const double C = 1.0 / (4.0 * 3.141592653589793238);
  T rx[4], ry[4], rz[4], R[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    rx[k] = T(rd_rec<SMEM>(rec + 3 * k) - q.x);
    ry[k] = T(rd_rec<SMEM>(rec + 3 * k + 1) - q.y);
    rz[k] = T(rd_rec<SMEM>(rec + 3 * k + 2) - q.z);
    R[k] = edge_R(rx[k], ry[k], rz[k]);
  }
  T d[6];  // r_i . r_j per edge
#pragma unroll
  for (int e = 0; e < 6; e++) {
    const int a = tet_edge_a(e), b = tet_edge_b(e);
    d[e] = rx[a] * rx[b] + ry[a] * ry[b] + rz[a] * rz[b];
  }
  double acc[TENSOR ? 6 : 3];
#pragma unroll
  for (int k = 0; k < (TENSOR ? 6 : 3); k++) acc[k] = 0.0;
  T Le[6];
  if constexpr (sizeof(T) == 8) {
    double S[6], l[6];
#pragma unroll
    for (int e = 0; e < 6; e++) {
      S[e] = R[tet_edge_a(e)] + R[tet_edge_b(e)];
      l[e] = rd_rec<SMEM>(rec + 12 + e);
    }
    edge_logs64<6>(S, l, Le, [&](int e) {
      const int a = tet_edge_a(e), b = tet_edge_b(e);
      return edge_D64(rx[a], ry[a], rz[a], R[a], rx[b], ry[b], rz[b], R[b]);
    });
  } else {
#pragma unroll
    for (int e = 0; e < 6; e++) {
      const int a = tet_edge_a(e), b = tet_edge_b(e);
      const T l = T(rd_rec<SMEM>(rec + 12 + e));
      Le[e] = edge_L(rx[a], ry[a], rz[a], R[a], rx[b], ry[b], rz[b], R[b], d[e], l);
    }
  }
#pragma unroll
  for (int e = 0; e < 6; e++) {
    const double L = (double)Le[e];
#pragma unroll
    for (int k = 0; k < (TENSOR ? 6 : 3); k++) acc[k] += L * rd_rec<SMEM>(rec + 42 + (TENSOR ? 6 : 3) * e + k);
  }
  double omega_tot = 0.0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    const int a = tet_face_a(f), b = tet_face_b(f), c = tet_face_c(f);
    const T m0 = T(rd_rec<SMEM>(rec + 18 + 3 * f));
    const T m1 = T(rd_rec<SMEM>(rec + 19 + 3 * f));
    const T m2 = T(rd_rec<SMEM>(rec + 20 + 3 * f));
    T num = rx[a] * m0 + ry[a] * m1 + rz[a] * m2;
    T den = R[a] * R[b] * R[c] + d[tet_pair(a, b)] * R[c] + d[tet_pair(a, c)] * R[b] + d[tet_pair(b, c)] * R[a];
    double om = 2.0 * (double)face_angle(-num, den);
    omega_tot += om;
    const double n0 = rd_rec<SMEM>(rec + 30 + 3 * f), n1 = rd_rec<SMEM>(rec + 31 + 3 * f), n2 = rd_rec<SMEM>(rec + 32 + 3 * f);
    if (TENSOR) {
      const double o0 = om * n0, o1 = om * n1, o2 = om * n2;
      acc[0] += o0 * n0; acc[1] += o0 * n1; acc[2] += o0 * n2;
      acc[3] += o1 * n1; acc[4] += o1 * n2; acc[5] += o2 * n2;
    } else {
      acc[0] += om * n0; acc[1] += om * n1; acc[2] += om * n2;
    }
  }
  if (TENSOR) {
    out[0] = C * acc[0];
    out[4] = C * acc[3];
    out[8] = C * acc[5];
    out[1] = out[3] = C * acc[1];
    out[2] = out[6] = C * acc[2];
    out[5] = out[7] = C * acc[4];
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++) out[k] = C * acc[k];
  }
  return omega_tot < -6.283185307179586;
}

}  // namespace rb
