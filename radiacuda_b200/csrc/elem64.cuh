// elem64.cuh -- FP64 square root, division, arctangent and logarithm of a
// ratio for the closed forms of the field sources.
//
// The closed forms are bound by the FP64 pipe (64 operations per clock and
// SM), and most of what they issue is the insides of sqrt, division, atan and
// log.  The library's versions treat every argument: subnormals, infinities,
// and a correctly rounded quotient.  Here the arguments are products of
// lengths, and a logarithm is always one of a ratio.  So these take a
// numerator and a denominator (one division for the argument reduction AND
// the ratio), positive normal arguments, and round to 1-2 ulp.
//
// Methods: reciprocal and reciprocal square root from the PTX approximations
// (rcp / rsqrt.approx.ftz.f64) by one step of Householder's third-order
// iteration, x (1 + e + e^2) and x (1 + e/2 + 3 e^2/8); the arctangent by the
// addition theorem with pi/4 and the logarithm as 2 artanh((n - d)/(n + d)),
// each a polynomial of least maximum relative error (Remez exchange) in the
// square of its argument.  tests/test_gpu_closed_forms.py holds the forms
// built on them against 64-bit references.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define RB_HD __host__ __device__ __forceinline__
#else
#define RB_HD inline
#endif

namespace rb {

// the two words of a double
RB_HD int hi32(double x)
{
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  int64_t b;
  memcpy(&b, &x, 8);
  return (int)(b >> 32);
#endif
}
RB_HD double add_hi32(double x, int d)  // x with d added to its upper word
{
#ifdef __CUDA_ARCH__
  return __hiloint2double(__double2hiint(x) + d, __double2loint(x));
#else
  int64_t b;
  memcpy(&b, &x, 8);
  b += (int64_t)((uint64_t)(uint32_t)d << 32);
  memcpy(&x, &b, 8);
  return x;
#endif
}
RB_HD double flip_sign(double x, int s)  // x, negated when s < 0
{
#ifdef __CUDA_ARCH__
  return __hiloint2double(__double2hiint(x) ^ (s & 0x80000000), __double2loint(x));
#else
  return s < 0 ? -x : x;
#endif
}

// 1 / d, d positive or negative normal
RB_HD double rcp64(double d)
{
  double y;
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
#else
  y = (1.0 / d) * (1.0 + 0x1p-20);  // the host check starts from an error of the approximation's size
#endif
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// sqrt(s), s positive normal
RB_HD double sqrt64(double s)
{
  double y;
#ifdef __CUDA_ARCH__
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
#else
  y = (1.0 / sqrt(s)) * (1.0 + 0x1p-20);
#endif
  const double g = s * y, e = fma(-g, y, 1.0);
  return fma(g * e, fma(0.375, e, 0.5), g);
}

// arctan(r) for |r| <= tan(pi/8): relative error of the polynomial 4.5e-18
RB_HD double atan_poly(double r)
{
  const double z = r * r;
  double p = -0x1.2431ee7ce89dfp-6;
  p = fma(p, z, 0x1.373c13fdd8fe9p-5);
  p = fma(p, z, -0x1.9c9123826d3cbp-5);
  p = fma(p, z, 0x1.deff55447b287p-5);
  p = fma(p, z, -0x1.10ea807e0ff11p-4);
  p = fma(p, z, 0x1.3b10fa21de456p-4);
  p = fma(p, z, -0x1.745cf6d8fb477p-4);
  p = fma(p, z, 0x1.c71c70d09c6e8p-4);
  p = fma(p, z, -0x1.2492492267e8fp-3);
  p = fma(p, z, 0x1.99999999948eep-3);
  p = fma(p, z, -0x1.5555555555531p-2);
  return fma(r * z, p, r);
}

// The angle of x + i y, plus 2 pi turns: sigma arctan(r) + j pi/4, |r| <=
// tan(pi/8), the quadrant and the turns collected in the integer j.
RB_HD double angle64(double y, double x, int turns)
{
  const double ax = fabs(x), ay = fabs(y);
  // compared by their upper words: the ranges only have to be met to 1e-5
  const bool swap = hi32(ay) > hi32(ax);
  const double mx = swap ? ay : ax, mn = swap ? ax : ay;
  const bool big = hi32(mn) > hi32(0.41421356237309503 * mx);
  const double c = big ? 1.0 : 0.0;
  const double a = atan_poly(fma(-c, mx, mn) * rcp64(fma(c, mn, mx)));
  int j = big ? 1 : 0, neg = 0;
  if (swap) { j = 2 - j; neg = ~neg; }
  if (hi32(x) < 0) { j = 4 - j; neg = ~neg; }
  if (hi32(y) < 0) { j = -j; neg = ~neg; }
  const double dj = (double)(j + 8 * turns);
  return fma(dj, 0.78539816339744828, fma(dj, 3.0616169978683830e-17, flip_sign(a, neg)));
}

// 2 artanh(s) = log((1 + s) / (1 - s)) for |s| <= 0.203: relative error of the
// polynomial 3.6e-17
RB_HD double artanh2_poly(double s)
{
  const double z = s * s;
  double p = 0x1.3c89e0ccdadebp-4;
  p = fma(p, z, 0x1.38143e890ab4dp-4);
  p = fma(p, z, 0x1.74783f2c7e313p-4);
  p = fma(p, z, 0x1.c71bea4baccf7p-4);
  p = fma(p, z, 0x1.249249db9161bp-3);
  p = fma(p, z, 0x1.99999998a73b4p-3);
  p = fma(p, z, 0x1.5555555555927p-2);
  const double t = s + s;
  return fma(t * z, p, t);
}
// k log(2) + L
RB_HD double add_klog2(int k, double L)
{
  const double dk = (double)k;
  return fma(dk, 0.69314718055994529, fma(dk, 2.3190468138462996e-17, L));
}
// both upper words those of normal numbers well inside the range
RB_HD bool plain_ratio(int hn, int hd)
{
  return (unsigned)(hn - 0x04000000) <= 0x78000000u && (unsigned)(hd - 0x04000000) <= 0x78000000u;
}

// log(n / d), n and d positive.  k: the power of two that brings n 2^-k / d
// into [0.66, 1.5], read off the upper words.  log_plain64: both of ordinary
// size (plain_ratio); log_ratio64 also takes zero, infinity and NaN (a point on
// an edge line), by the library's function.
RB_HD double log_plain64(double n, double d)
{
  const int k = (hi32(n) - hi32(d) + 0x80000) >> 20;
  const double m = add_hi32(n, -(k << 20));
  return add_klog2(k, artanh2_poly((m - d) * rcp64(m + d)));
}
RB_HD double log_ratio64(double n, double d) { return plain_ratio(hi32(n), hi32(d)) ? log_plain64(n, d) : log(n / d); }

// L = int dl / |q - r'| along an edge of length l, S = Ra + Rb the sum of its
// ends' distances from the point: log((S + l) / (S - l)) = 2 artanh(l / S),
// whose relative accuracy a distant point needs (the terms of a body cancel to
// third order there).  edge_log_far64: S - l not below S / 8.  Closer to the
// edge S - l cancels and is 2 D / (S + l), D = Ra Rb + a.b (edge_D64).  The
// two are apart so that a kernel can form several edges' far values without a
// branch between them and mend the rare near ones after.
RB_HD double edge_log_far64(double S, double l)
{
  const double n = S + l, d = S - l;
  const int k = (hi32(n) - hi32(d) + 0x80000) >> 20;
  const double m = add_hi32(n, -(k << 20));
  const double u = k ? m - d : l, v = k ? m + d : S;
  return add_klog2(k, artanh2_poly(u * rcp64(v)));
}
RB_HD bool edge_near64(double S, double l) { return hi32(S - l) < hi32(0.125 * S); }
#ifdef __CUDACC__
__host__ __device__ __noinline__ static
#else
static
#endif
double edge_log_near64(double S, double l, double D)
{
  const double n = S + l;
  return log_ratio64(n * n, 2.0 * D);
}
// D = Ra Rb + a.b of two offsets, |a x b|^2 / (Ra Rb - a.b) when a.b < 0
#ifdef __CUDACC__
__host__ __device__ __noinline__ static
#else
static
#endif
double edge_D64(double ax, double ay, double az, double Ra, double bx, double by, double bz, double Rb)
{
  const double s = fma(ax, bx, fma(ay, by, az * bz)), p = Ra * Rb;
  if (!(s < 0.0)) return p + s;
  const double cx = ay * bz - az * by, cy = az * bx - ax * bz, cz = ax * by - ay * bx;
  return (cx * cx + cy * cy + cz * cz) / (p - s);
}

// L of N edges, ends' distance sums S and lengths l: all far values first,
// then the near ones again; nearD(e) gives D of edge e
template <int N, typename F> RB_HD void edge_logs64(const double *S, const double *l, double *L, F nearD)
{
  bool near = false;
#pragma unroll
  for (int e = 0; e < N; e++) {
    L[e] = edge_log_far64(S[e], l[e]);
    near |= edge_near64(S[e], l[e]);
  }
  if (near) {
#pragma unroll
    for (int e = 0; e < N; e++)
      if (edge_near64(S[e], l[e])) L[e] = edge_log_near64(S[e], l[e], nearD(e));
  }
}

// arctan2(y, x)
RB_HD double atan2_64(double y, double x) { return angle64(y, x, 0); }

}  // namespace rb
