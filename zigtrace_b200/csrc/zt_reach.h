/*
 * zt_reach.h -- whether a hit point lies inside its primitive's box by more
 * than the f64 box test's rounding: the certainty the checked float walk
 * (zt_fast.cuh) needs of a hit.  Plain C++, so that the host can check it.
 */
#ifndef ZT_REACH_H
#define ZT_REACH_H

#include <math.h>

#if defined(__CUDACC__)
#define ZT_REACH_HD __host__ __device__ __forceinline__
#else
#define ZT_REACH_HD inline
#endif

namespace zt {

/* The margin asked for, per unit of M + |o| (M the largest bound, |o| the sum
 * of the origin's components).  What can go wrong on an axis, u = 2^-53: a
 * plane distance (b - o) * (1 / d) has three roundings, 3u (M + |o|) of
 * position; the point o + t d two, u (M + |o|) + u M; its offset from the
 * primitive, the primitive's extents, the sums below and the box's own
 * rounding at most 7u M: 12u (M + |o|) in all, of which this is 2.7 times. */
constexpr double kReachMargin = 0x1p-48;

/* One axis of a triangle's box: offset h of the point from the first vertex,
 * edges e1 and e2 to the others.  A box less than 1e-6 thick is padded by
 * 5e-7 on both sides (Aabb.pad, aabb.zig:30-39), which two edges below 2^-21
 * are certain to be. */
ZT_REACH_HD bool reach_triangle_axis(double h, double e1, double e2, double m) {
  const double s = (fabs(e1) < 0x1p-21) & (fabs(e2) < 0x1p-21) ? m - 4.95e-7 : m;
  const double lo = h - s, hi = h + s;
  return ((lo >= 0) | (lo >= e1) | (lo >= e2)) & ((hi <= 0) | (hi <= e1) | (hi <= e2));
}

/* a: first vertex and two edges, or centre and radius; (hx, hy, hz): the
 * point's offset from a[0..2]; m = kReachMargin * (M + |o|). */
ZT_REACH_HD bool reach_inside(bool triangle, const double* a, double hx, double hy, double hz, double m) {
  if (triangle)
    return reach_triangle_axis(hx, a[3], a[6], m) & reach_triangle_axis(hy, a[4], a[7], m) &
           reach_triangle_axis(hz, a[5], a[8], m);
  const double r = fabs(a[3]) - m;
  return (fabs(hx) <= r) & (fabs(hy) <= r) & (fabs(hz) <= r);
}

}  // namespace zt

#endif /* ZT_REACH_H */
