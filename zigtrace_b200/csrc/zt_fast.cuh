/*
 * zt_fast.cuh -- the float walk: the reference's BVH walk
 * (src/bvh.zig:80-126) over conservative single-precision boxes.
 *
 * The box tests of the f64 walk are three quarters of its arithmetic and run
 * on the FP64 pipe, which issues a warp instruction every other cycle per
 * SM sub-partition; their 128-byte pair records are most of its memory
 * traffic.  This walk tests the same tree's boxes in f32 (FMA, min/max) from
 * 64-byte records (FPair, zt_types.h) and keeps the primitive tests, the hit
 * records and all shading in f64, unchanged.
 *
 * Superset property.  A float box test here succeeds whenever the
 * reference's f64 test of the same box succeeds (same ray, same [tmin,
 * tmax]):
 *  - the ray is o + t d in f64; per axis the walk uses o32 = fl32(o),
 *    I = rcp(fl32(d)) (the hardware reciprocal, within 1 ulp, i.e. 2^-23
 *    relative; clamped to +-K, below) and n = fl32(-o32 I), and computes a
 *    plane distance as fl32(c I + off) with one FMA, c the float plane and
 *    off = n -+ w.  Against the exact (c - o) / d the error is at most
 *    2^-23 (2 |c| + 3.5 |o|) / |d| (rounding of d, of o, of the product n,
 *    of the FMA and of n -+ w, each at most 2^-24 relative, and the
 *    reciprocal's 2^-23);
 *  - the |c| part is covered by the records: every bound is moved outward by
 *    eps = 2^-20 M (M the largest |bound| on that axis; 4x the 2 2^-23 M
 *    needed; kFastMinMargin at least), which moves a near plane's distance
 *    down and a far plane's up by eps / |d|;
 *  - the |o| part is covered per ray: w = 2^-20 |n| (2.3x the 3.5 2^-23 |o I|
 *    needed) is subtracted from near planes and added to far planes;
 *  - so each near distance is at most the exact one and each far distance at
 *    least the exact one, tmin is rounded down and tmax up, and an interval
 *    the exact test finds non-empty stays non-empty.  The f64 test's own
 *    rounding (2^-53 relative) is far inside these margins.
 *  - A zero or tiny direction component has its reciprocal clamped to +-K
 *    with K |o| <= 1e37 and K M <= 1e37 (M <= kFastMaxCoord), so no product
 *    overflows.  Near distances only get smaller by that (in magnitude where
 *    the ray starts outside the slab, in sign where it starts inside).  The
 *    far distance does too, and must still exceed every distance t at which
 *    the ray can be in the slab: it is at least 3/4 K eps - t (eps the
 *    record's margin, of which the roundings above take at most a quarter;
 *    a component below 1/K moves the ray by at most t/K on the axis), so
 *    3/4 K eps >= 2 t is needed.  The scene's bounds end at t <= 1.8 (|o| +
 *    1.8 M) / |d|, |d| >= 0.28 (fray_make).  For |o| <= 1e7 that is 2e8, and
 *    3/4 K eps >= 7e14 (K = 1e30, eps >= kFastMinMargin).  Beyond, K = 1e37 /
 *    |o| falls as t rises: at kFastMaxOrigin = 1e10, t <= 6.5e10 and 3/4 K eps
 *    >= 7e11.  (At the 1e30 this limit once was, a box straight ahead of a
 *    ray parallel to an axis was missed from about 3e18 on, and from less in
 *    flat scenes.)
 * Entry distances are lower bounds of the exact ones, so `entry.t > closest`
 * against closest rounded up drops a node only when the ray enters its box
 * behind a hit already found, and leaves are tested with the reference's f64
 * primitive tests.  The closest hit found is therefore the least primitive
 * distance over a superset of the leaves the reference tests; it differs from
 * the reference's only
 *  - where two primitives tie;
 *  - where the reference's own f64 box test misses a primitive hit by rounding
 *    (a grazing ray);
 *  - where a primitive in a dropped node is hit in front of its own box, and the
 *    reference, which may come to that node before the other hit, tests it.
 *    The boxes' margins (2^-20 of the coordinates) exceed what a sphere test
 *    errs by; a triangle's distance errs by 18u (|s| + |e|) |e1||e2| / |det|
 *    (light_passed in zt_device.cuh), more than the margins only where the ray
 *    meets the triangle at a cosine below some 2e-9 |e1||e2| / |e1 x e2|.
 * ZT_PRECISION_FAST takes the result as it is: its images are held to a
 * statistical bar (per-channel relative RMSE and mean luminance against the
 * oracle), not to bit equality.
 *
 * The checked walk (kVerify, ZT_PRECISION_EXACT) detects the first two, so its
 * results are the f64 walk's bit for bit but for the third, which is not
 * detected and has not been met (a ray within 2e-9 of a triangle's plane, and
 * another hit within the error of it):
 *  - a tie: another primitive is hit at exactly the closest distance.  In
 *    one leaf both walks test the primitives in the same order and the first
 *    keeps the hit (coincident primitives have one centroid, which no split
 *    separates); between two leaves the f64 walk's order of visiting them is
 *    worked out (tie_first); a third primitive at the distance leaves a doubt.
 *    With every tie in doubt, the 250k-triangle terrain 961x541x16 with each
 *    fiftieth triangle twice took 22.6 ms, now 10.6, with the f64 walk alone
 *    14.0; a closed box of 2,572 triangles with its light in the plane of its
 *    ceiling, 800x800x32, 122 ms, 40.2 and 39.8;
 *  - a hit whose leaf the f64 walk might miss: walk_reaches shows that the
 *    hit point lies inside the primitive's box by more than the f64 test's
 *    rounding.  Every ancestor's box holds that box (boxes_nested), so the
 *    f64 test passes at every node on the way down, and no entry distance
 *    exceeds the hit's, so no pop is pruned: the f64 walk tests the
 *    primitive, and it is the least hit of a superset of what that walk
 *    tests (the third case apart).  No hit in the superset means none in the
 *    f64 walk: nothing is dropped before a first hit.
 * Where either is in doubt `doubt` is set and the caller renders the pixel
 * again with the f64 walk (none of the images measured below: the flag costs
 * a register, where a call of the f64 walk from inside this one measured 7% on
 * the 1M-triangle terrain and 12% on the sphere fields).  Rays the float
 * test does not take (fray_make) go the same way.  The margin walk_reaches
 * asks for is derived in zt_reach.h.  It is compared in f64: in single
 * precision the extents' rounding had to be allowed for (2^-20 of them), which
 * left the middle of a ground made of a large sphere in doubt, 1.4 units
 * around the pole at radius 1000: of random spheres on such a ground
 * (1280x720x16) 2.7% of the pixels were rendered twice, and the image took
 * 7.3 ms, now 3.85, with the f64 walk alone 5.6; at radius 5000 55%, 12.0 ms,
 * 3.87 and 5.6.  The f64 comparisons also take less time than the conversions
 * did (random spheres 3.78 -> 3.61 ms, terrain unchanged).
 * Measured, against the f64 walk with its 128-byte records: 250k-triangle
 * terrain 961x541x16 15.0 -> 11.2 ms, random spheres 1280x720x16 5.34 ->
 * 3.75 ms, 256 sphere fields 71.9 -> 51.9 ms.
 *
 * Stack entries are 8 bytes (packed payload word + float entry distance),
 * 4 bytes in the any-hit walk.
 */
#ifndef ZT_FAST_CUH
#define ZT_FAST_CUH

#include "zt_reach.h"

namespace zt {

/* Per-ray constants of the float slab test, as packed f32x2 operands: per
 * axis the reciprocal twice, and the offsets of the planes through a box's
 * lower and upper bound (the FPair layout's order). */
struct FRay {
  unsigned long long inv2[3];
  unsigned long long off2[3];
};

ZT_D unsigned long long f2_pack(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
/* Both plane distances of one axis: fl32(c * inv + off) for c = lower and
 * upper bound, each lane one FMA with a single rounding (as fmaf). */
ZT_D void f2_planes(unsigned long long box, unsigned long long inv2, unsigned long long off2, float& a, float& b) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(box), "l"(inv2), "l"(off2));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
/* Three-input minimum and maximum (sm_100). */
ZT_D float fmax3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
ZT_D float fmin3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

/* Largest |origin| (component sum) the float test takes (derived above).
 * Rays from farther away (a hit far out on an unbounded plane), with a NaN, or
 * with a direction far from unit length leave the pixel in doubt. */
constexpr float kFastMaxOrigin = 1e10f;

ZT_D bool fray_make(dv3 o, dv3 d, FRay& r) {
  const float o3[3] = {(float)o.x, (float)o.y, (float)o.z};
  const float d3[3] = {(float)d.x, (float)d.y, (float)d.z};
  const float om = fmaxf(fabsf(o3[0]), fmaxf(fabsf(o3[1]), fabsf(o3[2])));
  const float os = fabsf(o3[0]) + fabsf(o3[1]) + fabsf(o3[2]); /* sums: a NaN component fails the test */
  const float ds = fabsf(d3[0]) + fabsf(d3[1]) + fabsf(d3[2]);
  if (!(os <= kFastMaxOrigin && ds >= 0.5f && ds <= 2.0f)) return false; /* ds: 1 to sqrt(3) of a unit vector */
  const float K = om > 1e7f ? 1e37f / om : 1e30f; /* K |o| <= 1e37, K * kFastMaxCoord <= 1e37 */
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(d3[a])); /* within 1 ulp; +-0 (and flushed subnormals) give +-inf */
    if (!(fabsf(inv) <= K)) inv = copysignf(K, inv); /* +-inf (a zero component) and huge values */
    const float n = -o3[a] * inv;
    const float w = fabsf(n) * 0x1.0p-20f;
    /* lower plane nearer when inv >= 0: it takes n - w, the upper plane n + w */
    r.inv2[a] = f2_pack(inv, inv);
    r.off2[a] = inv >= 0.0f ? f2_pack(n - w, n + w) : f2_pack(n + w, n - w);
  }
  return true;
}

/* Float slab test of one box given as its three (lower, upper) axis pairs;
 * tnear is the (lower-bound) entry distance. */
ZT_D bool fslab(unsigned long long bx, unsigned long long by, unsigned long long bz, const FRay& r, float tmin,
                float tmax, float& tnear) {
  float a0, b0, a1, b1, a2, b2;
  f2_planes(bx, r.inv2[0], r.off2[0], a0, b0);
  f2_planes(by, r.inv2[1], r.off2[1], a1, b1);
  f2_planes(bz, r.inv2[2], r.off2[2], a2, b2);
  const float n = fmax3f(fminf(a0, b0), fminf(a1, b1), fmaxf(fminf(a2, b2), tmin));
  const float f = fmin3f(fmaxf(a0, b0), fmaxf(a1, b1), fminf(fmaxf(a2, b2), tmax));
  tnear = n;
  return n <= f;
}

/* Whether the f64 walk is certain to reach the leaf of primitive p, hit at
 * `point` by a ray from o: the point is inside the primitive's box by the
 * margin derived in zt_reach.h. */
ZT_D bool walk_reaches(const DevScene& sc, const DPrim& p, dv3 o, dv3 point) {
  const double m = kReachMargin * ((double)sc.freach + fabs(o.x) + fabs(o.y) + fabs(o.z));
  const dv3 h = point - L3(p.a);
  return reach_inside(p.kind == kTriangle, p.a, h.x, h.y, h.z, m);
}

/* Which of two primitives of different leaves, a and b, hit at the same
 * distance t, the f64 walk tests first and so keeps; -1 where that cannot be
 * shown.  Both hits must be certain to be reached (walk_reaches); the walk then
 * enters both children of the lowest node above the two leaves, the nearer one
 * first, and finishes with it before the other.  The node is found from the
 * root by the records' splits, and its children's entry distances are the f64
 * walk's own (slab).  A call, and its result by value: inlined, random spheres
 * took 4.00 ms against 3.86. */
__device__ __noinline__ int32_t tie_first(const DevScene& sc, dv3 o, dv3 d, double tmin, double t, int32_t a,
                                          int32_t b) {
  const dv3 point = o + vscale(d, t);
  if (!walk_reaches(sc, sc.prims[a], o, point) || !walk_reaches(sc, sc.prims[b], o, point)) return -1;
  uint32_t w = sc.froot_word;
  bool a_right;
  for (;;) {
    if (w >> kFastCountShift) return -1; /* no order to go by (kNoSplit) */
    const FPair& r = sc.fpairs[w];
    a_right = (uint32_t)a >= r.split;
    if (a_right != ((uint32_t)b >= r.split)) break;
    w = r.word[a_right];
  }
  const DPair& p = sc.pairs[w];
  const dv3 inv = V(1.0 / d.x, 1.0 / d.y, 1.0 / d.z);
  double tl, tr;
  slab(p.lo[0], p.hi[0], o, inv, tmin, t, tl);
  slab(p.lo[1], p.hi[1], o, inv, tmin, t, tr);
  return (tl <= tr) != a_right ? a : b;
}

/* One 64-byte record: both children's axis pairs and payload words. */
struct FRec {
  ulonglong2 q0, q1, q2;
  uint2 w;
};
ZT_D FRec frec_load(const FPair* p) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(p);
  FRec r;
  r.q0 = __ldg(q);
  r.q1 = __ldg(q + 1);
  r.q2 = __ldg(q + 2);
  r.w = __ldg(reinterpret_cast<const uint2*>(q + 3));
  return r;
}
/* left x y = q0.x q0.y, left z = q1.x; right x = q1.y, right y z = q2.x q2.y */
ZT_D bool fslab_left(const FRec& r, const FRay& fr, float tmin, float tmax, float& t) {
  return fslab(r.q0.x, r.q0.y, r.q1.x, fr, tmin, tmax, t);
}
ZT_D bool fslab_right(const FRec& r, const FRay& fr, float tmin, float tmax, float& t) {
  return fslab(r.q1.y, r.q2.x, r.q2.y, fr, tmin, tmax, t);
}
ZT_D bool fslab_root(const DevScene& sc, const FRay& fr, float tmin, float tmax, float& t) {
  return fslab(f2_pack(sc.froot[0][0], sc.froot[0][1]), f2_pack(sc.froot[1][0], sc.froot[1][1]),
               f2_pack(sc.froot[2][0], sc.froot[2][1]), fr, tmin, tmax, t);
}

/* Scene.intersect (scene.zig:108-116) with the BVH walked over the float
 * records: nearest first by float entry distance (ties to the left child,
 * bvh.zig:111-116), pruning entries whose distance exceeds the closest hit,
 * f64 primitive tests; then the unbounded planes.  Return value and t_out as
 * scene_query_rt's (closest hit only).  kVerify notes what is in doubt (0:
 * nothing, k + 1: primitive k ties with the hit, -1: the f64 walk has to
 * decide); the caller checks the hit itself with walk_reaches, beside its hit
 * record. */
template <bool kVerify>
ZT_D int32_t scene_query_fast(const DevScene& sc, dv3 o, dv3 d, double tmin, double tmax, double& t_out,
                              int32_t& doubt) {
  double closest = tmax;
  int32_t best_k = -1;
  if (sc.has_root) {
    FRay fr;
    if (!fray_make(o, d, fr)) {
      doubt = -1;
      return -1;
    }
    const float tmin32 = __double2float_rd(tmin);
    float cl32 = __double2float_ru(closest);
    float t;
    if (fslab_root(sc, fr, tmin32, cl32, t)) {
      uint2 stack[kStackSize]; /* (payload word, entry distance bits) */
      uint32_t w = sc.froot_word;
      float et = t;
      bool have = true;
      int sp = 0;
      for (;;) {
        if (!have) {
          if (sp == 0) break;
          const uint2 e = stack[--sp];
          w = e.x;
          et = __uint_as_float(e.y);
        }
        have = false;
        if (et > cl32) continue; /* bvh.zig:97, against closest rounded up */
        const uint32_t cnt = w >> kFastCountShift, first = w & kFastFirstMask;
        if (cnt > 0) {
          /* One word counts the leaf's primitives off and holds the next one's index; in a leaf a hit of its own is
           * kept as -2 - k.  (With an end index the 256 sphere fields took 52.6 ms, so 51.9, with
           * ZT_PRECISION_FAST 51.3 and 50.5.) */
          uint32_t left = w;
          do {
            const uint32_t k = left & kFastFirstMask;
            double th;
            if (bounded_t<kVerify>(sc.prims[k], o, d, tmin, closest, th)) {
              if (kVerify && !(th < closest)) {
                /* a tie (or a NaN): in one leaf the first primitive keeps the hit, as in the f64 walk; between
                 * leaves that walk's visiting order decides (tie_first) */
                if (best_k >= -1 || !(th == closest))
                  doubt = best_k >= 0 && th == closest && doubt == 0 ? (int32_t)k + 1 : -1;
              } else {
                closest = th;
                best_k = kVerify ? -2 - (int32_t)k : (int32_t)k;
                cl32 = __double2float_ru(th);
                if (kVerify) doubt = min(doubt, 0); /* ties behind the hit are of no account */
              }
            }
            left += 1u - (1u << kFastCountShift);
          } while (left >> kFastCountShift);
          if (kVerify && best_k < -1) best_k = -2 - best_k;
          continue;
        }
        const FRec r = frec_load(sc.fpairs + first);
        float tl, tr;
        const bool hl = fslab_left(r, fr, tmin32, cl32, tl);
        const bool hr = fslab_right(r, fr, tmin32, cl32, tr);
        if (hl && hr) { /* push the farther child; the nearer one is next */
          const bool near_left = tl <= tr;
          stack[sp] = make_uint2(near_left ? r.w.y : r.w.x, __float_as_uint(near_left ? tr : tl));
          sp += 1;
          w = near_left ? r.w.x : r.w.y;
          et = near_left ? tl : tr;
          have = true;
        } else if (hl || hr) {
          w = hl ? r.w.x : r.w.y;
          et = hl ? tl : tr;
          have = true;
        }
      }
    }
  }
  for (uint32_t i = 0; i < sc.n_planes; ++i) { /* geometry.zig:129-139 */
    double th;
    if (plane_prim_t(sc.planes[i], o, d, tmin, closest, th)) {
      closest = th;
      best_k = -2 - (int32_t)i;
      if (kVerify) doubt = min(doubt, 0);
    }
  }
  t_out = closest;
  return best_k;
}

/* Shadow query over the float records: whether any primitive is hit in
 * (tmin, tmax).  The leaves it tests are a superset of the leaves the f64
 * walk tests, and any primitive hit below tmax is an occluder whichever walk
 * finds it; kVerify checks that the f64 walk reaches the one found.  Farther
 * child first, as scene_occluded. */
template <bool kVerify>
ZT_D bool scene_occluded_fast(const DevScene& sc, dv3 o, dv3 d, double tmin, double tmax, int32_t& doubt) {
  if (sc.has_root) {
    FRay fr;
    if (!fray_make(o, d, fr)) {
      doubt = -1;
      return true;
    }
    const float tmin32 = __double2float_rd(tmin), tmax32 = __double2float_ru(tmax);
    float t;
    if (fslab_root(sc, fr, tmin32, tmax32, t)) {
      uint32_t stack[kStackSize];
      uint32_t w = sc.froot_word;
      bool have = true;
      int sp = 0;
      for (;;) {
        if (!have) {
          if (sp == 0) break;
          w = stack[--sp];
        }
        have = false;
        const uint32_t cnt = w >> kFastCountShift, first = w & kFastFirstMask;
        if (cnt > 0) {
          for (uint32_t k = first; k < first + cnt; ++k) {
            double th;
            if (prim_t(sc.prims[k], o, d, tmin, tmax, th)) {
              if (kVerify && !walk_reaches(sc, sc.prims[k], o, o + vscale(d, th))) doubt = -1;
              return true;
            }
          }
          continue;
        }
        const FRec r = frec_load(sc.fpairs + first);
        float tl, tr;
        const bool hl = fslab_left(r, fr, tmin32, tmax32, tl);
        const bool hr = fslab_right(r, fr, tmin32, tmax32, tr);
        if (hl && hr) {
          const bool left_first = tl > tr; /* the farther child first */
          stack[sp++] = left_first ? r.w.y : r.w.x;
          w = left_first ? r.w.x : r.w.y;
          have = true;
        } else if (hl || hr) {
          w = hl ? r.w.x : r.w.y;
          have = true;
        }
      }
    }
  }
  for (uint32_t i = 0; i < sc.n_planes; ++i) {
    double th;
    if (prim_t(sc.planes[i], o, d, tmin, tmax, th)) return true;
  }
  return false;
}

}  // namespace zt

#endif
