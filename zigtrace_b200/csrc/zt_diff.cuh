/*
 * zt_diff.cuh -- the differentiable form of traceWith: gradients of an image
 * loss with respect to every material's colour (the albedo of Lambertian and
 * metal materials, the radiance of emissive ones).
 *
 * Detached sampling.  The scene's own materials (theta0) drive every sampling
 * decision: the roulette probability comes from a throughput built with
 * theta0's albedos, the light pick from the theta0 emitter table, and the MIS
 * weights from theta0's pdfs.  Contributions are evaluated with the parameters
 * theta.  Each sample is then a product of parameter factors times constants
 * fixed by the random numbers, so with common random numbers it is a smooth
 * function of theta, and its expectation is the rendering at theta (an
 * importance-sampled estimator with a fixed proposal is unbiased).  At
 * theta == theta0 every operation is traceWith's (render.zig:61-102) in the
 * same order, so the image is the reference image bit for bit.
 *
 * Path replay.  The adjoint of one sample re-runs its path from the saved RNG
 * state (no tape).  A scatter at material m multiplies every term added
 * after it by theta[m], so d/d theta[m] gets adj * (L - R) / theta[m], with L
 * the sample's radiance (from the primal pass) and R the radiance added so
 * far; emission and light-sample terms add their own direct derivatives.
 * A zero albedo channel contributes no gradient (the proposal never
 * continues a path past it).
 */
#ifndef ZT_DIFF_CUH
#define ZT_DIFF_CUH

#include "zt_device.cuh"

namespace zt {

/* Adds v to grad[3m..3m+2], in global memory without a returned value: the
 * warp issues three instructions and goes on, and the L2 does the additions.
 * (Lanes adding in turn to the warp's slice in shared memory kept the warp
 * for a load, an add and a store per active lane: the backward took 50.0 ms
 * that way and 39.6 with this, both without regeneration.) */
ZT_D void grad_add(double* grad, uint32_t m, dv3 v) {
  double* q = grad + 3 * (size_t)m;
  atomicAdd(q + 0, v.x);
  atomicAdd(q + 1, v.y);
  atomicAdd(q + 2, v.z);
}

/* The BVH query as a real call: the differentiable kernels are instruction-
 * cache bound when each of their queries inlines its own copy of the
 * traversal (measured: forward and backward ~22% faster outlined).  One
 * function for closest hits and shadow rays, told apart at run time, for the
 * same reason: with a second one for shadow rays the forward took 31.2 ms
 * against 25.3 (512x512x64), the backward 35.4 against 28.8. */
__device__ __noinline__ int32_t scene_query_outlined(const DevScene& sc, dv3 o, dv3 d, double tmin, double tmax,
                                                     bool any_hit, double& t_out) {
  return scene_query_rt(sc, o, d, tmin, tmax, any_hit, t_out);
}

/* A path between two bounces. */
struct DiffPath {
  dv3 ro, rd, radiance, tp, tp0; /* tp with theta, tp0 with theta0 (the roulette's) */
  double prev_pdf;
};
ZT_D void diff_start(DiffPath& s) {
  s.radiance = V(0, 0, 0);
  s.tp = s.tp0 = V(1, 1, 1);
  s.prev_pdf = 0;
}

/* One iteration of traceWith's bounce loop; true when the path has ended.
 * kAdj is a run-time flag so that the primal and the replay pass of the
 * backward kernel share one copy of this code (the kernel is instruction-
 * cache bound with two copies).  prev_origin (render.zig:66-70) is read only
 * after a bounce, where it equals ro: ro stands in for it, as in trace_with.
 * Both derivatives with respect to the hit's own colour, the light sample's
 * and that of every later term, are added at once. */
ZT_D bool diff_bounce(const DevScene& sc, const double* __restrict__ theta, DiffPath& s, uint64_t depth, Rng& rng,
                      bool use_nee, bool kAdj, dv3 L_total, dv3 adj, double* grad) {
  Hit hit;
  double th_t;
  const int32_t hk = scene_query_outlined(sc, s.ro, s.rd, kRayEpsilon, INFINITY, false, th_t);
  if (hk == -1) {
    s.radiance = s.radiance + vmul(s.tp, background_radiance(sc.bg, s.rd));
    return true;
  }
  hit_from(sc, hk, s.ro, s.rd, th_t, hit);
  const uint32_t m = hit.material;
  const DMat& mat = sc.mats[m];
  const dv3 th = L3(theta + 3 * (size_t)m);
  const bool emits = mat.kind == kEmissive && hit.front_face;
  const dv3 le0 = emits ? L3(mat.color) : V(0, 0, 0);
  if (vmaxc(le0) > 0) { /* emission with its MIS weight, render.zig:77-81 */
    const double w = s.prev_pdf > 0 ? power_weight(s.prev_pdf, lights_pdf_hit(sc, s.ro, hit.point)) : 1.0;
    if (kAdj) grad_add(grad, m, vmul(adj, vscale(s.tp, w)));
    s.radiance = s.radiance + vscale(vmul(s.tp, th), w);
  }
  dv3 own = V(0, 0, 0); /* d/d theta[m] of the light sample and of what follows, without adj */
  if (mat.kind == kLambertian && use_nee) { /* directLight, render.zig:46-56 */
    dv3 ldir, lrad0, direct = V(0, 0, 0);
    double ldist, lpdf;
    uint32_t li = 0;
    if (lights_sample(sc, hit.point, rng, ldir, ldist, lrad0, lpdf, &li)) {
      const double cos_s = vdot(hit.normal, ldir);
      if (!(cos_s <= 0 || !(lpdf > 0))) {
        double st;
        if (scene_query_outlined(sc, hit.point, ldir, kRayEpsilon, ldist * (1 - 1e-6), true, st) == -1) {
          const double bsdf_pdf = cos_s / kPi;
          const double scale = cos_s / (kPi * lpdf) * power_weight(lpdf, bsdf_pdf);
          const uint32_t lm = sc.lights[li].material;
          const dv3 lrad = L3(theta + 3 * (size_t)lm);
          direct = vscale(vmul(th, lrad), scale);
          if (kAdj) {
            own = vscale(vmul(s.tp, lrad), scale);
            grad_add(grad, lm, vmul(adj, vscale(vmul(s.tp, th), scale)));
          }
        }
      }
    }
    s.radiance = s.radiance + vmul(s.tp, direct);
  }
  dv3 atten0, sd;
  const bool scattered = material_scatter(mat, s.rd, hit, rng, atten0, sd);
  const bool param = mat.kind == kLambertian || mat.kind == kMetal;
  if (kAdj && param) { /* every later term carries theta[m]: their sum is L_total - radiance */
    if (scattered) {
      const dv3 rest = L_total - s.radiance;
      own = own + V(th.x != 0 ? rest.x / th.x : 0.0, th.y != 0 ? rest.y / th.y : 0.0, th.z != 0 ? rest.z / th.z : 0.0);
    }
    grad_add(grad, m, vmul(adj, own));
  }
  if (!scattered) return true;
  s.tp = vmul(s.tp, param ? th : atten0);
  s.tp0 = vmul(s.tp0, atten0);
  s.prev_pdf = (use_nee && mat.kind == kLambertian) ? fmax(vdot(sd, hit.normal), 0.0) / kPi : 0;
  s.ro = hit.point;
  s.rd = sd;
  if (depth + 1 >= kRouletteDepth) { /* roulette on the theta0 throughput */
    const double p = fmin(vmaxc(s.tp0), 0.95);
    if (p <= 0 || rng_float(rng) >= p) return true;
    s.tp = vdiv(s.tp, p);
    s.tp0 = vdiv(s.tp0, p);
  }
  return false;
}

}  // namespace zt

#endif
