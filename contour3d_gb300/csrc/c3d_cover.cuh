/*
 * c3d_cover.cuh -- FP32 areas, edge functions and weights of a screen triangle
 * with certified bounds: k_emit's area rule and the coverage test of k_raster.
 * Plain float arithmetic (fused only where __fmaf_rn says so), with kU32 =
 * 2^-24 and `eps` the bound on a vertex's distance to the reference's.
 */
#pragma once

namespace c3d {

struct EdgeF {
  float ax, ay, dby, dbx, e_dby, e_dbx;
};

__device__ __forceinline__ EdgeF edge_f(float ax, float ay, float bx, float by, float eps) {
  EdgeF E;
  E.ax = ax;
  E.ay = ay;
  E.dby = by - ay;
  E.dbx = bx - ax;
  E.e_dby = 2.f * eps + kU32 * fabsf(E.dby);
  E.e_dbx = 2.f * eps + kU32 * fabsf(E.dbx);
  return E;
}

/* render.c:38-46 at a point known to +-e_p, edge vertex a known to +-eps_a; value and error bound */
__device__ __forceinline__ float edge_eval(const EdgeF& E, float px, float py, float e_p, float eps_a, float& err) {
  const float u = px - E.ax, v = py - E.ay;
  const float eu = __fmaf_rn(kU32, fabsf(u), e_p + eps_a), ev = __fmaf_rn(kU32, fabsf(v), e_p + eps_a);
  /* u dby - v dbx with one rounding of the product v dbx and one of the
     fused result; the bound keeps a term for a rounding of u dby as well */
  const float p2 = v * E.dbx;
  const float e = __fmaf_rn(u, E.dby, -p2);
  const float pr = fabsf(u) * fabsf(E.dby) + fabsf(p2) + fabsf(e);
  float b = __fmaf_rn(fabsf(u), E.e_dby, kU32 * pr);
  b = __fmaf_rn(fabsf(E.dby) + E.e_dby, eu, b);
  b = __fmaf_rn(fabsf(v), E.e_dbx, b);
  b = __fmaf_rn(fabsf(E.dbx) + E.e_dbx, ev, b);
  err = 1.25f * b;
  return e;
}

/* the area (render.c:38-46) as edge_eval computes it, with its bound in the
   factored form: every difference is off by at most 2 exy and a rounding */
__device__ __forceinline__ float emit_area(const float X[3], const float Y[3], float exy, float& errA) {
  const float dbx = X[1] - X[0], dby = Y[1] - Y[0], u = X[2] - X[0], w = Y[2] - Y[0];
  const float p2 = w * dbx;
  errA = __fmaf_rn(2.5f * exy, __fmaf_rn(4.f, exy, (fabsf(u) + fabsf(w)) + (fabsf(dbx) + fabsf(dby))),
                   5.f * kU32 * (fabsf(u * dby) + fabsf(p2)));
  return __fmaf_rn(u, dby, -p2);
}

/* an area that the reference certainly does not clamp to +-1e-16 (render.c:108-111) */
__device__ __forceinline__ bool area_unclamped(float A, float errA) { return fabsf(A) - errA > 1e-15f; }

constexpr float kWOut = -1.0e-8f * (1.f + 1e-5f); /* certainly below -1e-8 */
constexpr float kWIn = -1.0e-8f * (1.f - 1e-5f);  /* certainly above -1e-8 */

/* a cover-list triangle's edges, area and inverse area (render.c:102-107) with
   bounds; k_emit listed only triangles whose area is certainly not clamped.
   The weight bounds are used when they are tight enough to decide anything
   (rai < 0.5) */
struct CoverTri {
  EdgeF E0, E1, E2;
  float eps, ai, rai;
};

__device__ __forceinline__ CoverTri cover_tri(const float X[3], const float Y[3], float eps) {
  CoverTri c;
  c.E0 = edge_f(X[1], Y[1], X[2], Y[2], eps);
  c.E1 = edge_f(X[2], Y[2], X[0], Y[0], eps);
  c.E2 = edge_f(X[0], Y[0], X[1], Y[1], eps);
  c.eps = eps;
  float errA;
  const float A = edge_eval(c.E2, X[2], Y[2], eps, eps, errA);
  /* this bound's roundings are not emit_area's: it may reach |A|, and then decides
     nothing.  |A| is below 1e10 on any screen: __fdividef is within 2 ulp */
  const float room = fabsf(A) - errA;
  c.rai = room > 0.f ? 1.001f * __fdividef(errA, room) + 6.f * kU32 : INFINITY;
  c.ai = __fdividef(1.f, A);
  return c;
}

/* the pixel centre (px, py) certainly outside (out) or certainly inside the triangle */
__device__ __forceinline__ void cover_test(const CoverTri& c, float px, float py, bool& out, bool& inside) {
  const float ep = 0.5f * kU32;
  float e0, e1, e2;
  const float w0 = c.ai * edge_eval(c.E0, px, py, ep, c.eps, e0);
  const float w1 = c.ai * edge_eval(c.E1, px, py, ep, c.eps, e1);
  const float w2 = c.ai * edge_eval(c.E2, px, py, ep, c.eps, e2);
  const float k = fabsf(c.ai) * (1.f + c.rai), kr = c.rai + kU32;
  const float ew0 = __fmaf_rn(1.25f, __fmaf_rn(k, e0, fabsf(w0) * kr), 1e-30f);
  const float ew1 = __fmaf_rn(1.25f, __fmaf_rn(k, e1, fabsf(w1) * kr), 1e-30f);
  const float ew2 = __fmaf_rn(1.25f, __fmaf_rn(k, e2, fabsf(w2) * kr), 1e-30f);
  const bool ok = c.rai < 0.5f;
  out = ok && ((w0 + ew0 < kWOut) || (w1 + ew1 < kWOut) || (w2 + ew2 < kWOut));
  inside = ok && !out && (w0 - ew0 > kWIn) && (w1 - ew1 > kWIn) && (w2 - ew2 > kWIn);
}

}  // namespace c3d
