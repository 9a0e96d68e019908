// Quadrature tiers of the periodic domain's regular pairs: which of the
// shorter rules an element takes at a given distance from a source of the
// Green's function's singularity, and that rule's points.
#pragma once
#include "bem_geom.cuh"

__device__ __forceinline__ double tier_dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
// the quad's shape guard of tiers 0, 1, 3 and 4: the part of its twist c3
// along the normal c1 x c2 at most a tenth of its shorter half-side |c1| or
// |c2|, and the longer half-side at most 3 times the shorter
__device__ __forceinline__ bool quad_tier_shape(const bem_el &el) {
  double c1[3], c2[3], c3[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) { c1[d] = el.cr[d][1]; c2[d] = el.cr[d][2]; c3[d] = el.cr[d][3]; }
  const double n0 = c1[1] * c2[2] - c1[2] * c2[1], n1 = c1[2] * c2[0] - c1[0] * c2[2], n2 = c1[0] * c2[1] - c1[1] * c2[0];
  const double nn = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
  const double l1 = sqrt(tier_dot3(c1, c1)), l2 = sqrt(tier_dot3(c2, c2));
  const double lmin = fmin(l1, l2), lmax = fmax(l1, l2);
  return nn > 0.0 && fabs(c3[0] * n0 + c3[1] * n1 + c3[2] * n2) <= 0.1 * lmin * nn && lmax <= 3.0 * lmin;
}
// squared circumradius of the element about its centre (a triangle's centroid)
__device__ __forceinline__ double el_circum2(const bem_el &el, bool tri) {
  // corners (+-1, +-1) of a quad, (1, 0), (-1/2, +-sqrt3/2) of a triangle
  double R2 = 0.0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double sz = (c == 1 || c == 2) ? 1.0 : -1.0, se = c >= 2 ? 1.0 : -1.0;
    if (tri) {
      sz = c == 0 ? 1.0 : -0.5;
      se = c == 0 ? 0.0 : (c == 1 ? 0.5 * BEM_SQ3 : -0.5 * BEM_SQ3);
    }
    double v2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double v = el.cr[d][1] * sz + el.cr[d][2] * se + el.cr[d][3] * sz * se;
      v2 += v * v;
    }
    R2 = fmax(R2, v2);
  }
  return R2;
}
// tier for a singularity at r2 = (distance / R)^2 from the element's centre and
// kR2 = (k R)^2; -1: the reference's 12 x 12 rule
__device__ __forceinline__ int tier_of(double r2, double kR2, bool tri, bool shape) {
  if (kR2 > 1.0) return -1;
  if (tri)  // flat triangles converge faster: 7 points from 6 R, 6 from 12 R (k R <= 0.5)
    return r2 >= 144.0 && kR2 <= 0.25 ? 4 : r2 >= 36.0 && kR2 <= 0.25 ? 3 : r2 >= 25.0 ? 2 : r2 >= 12.25 ? 1 : r2 >= 9.0 ? 0 : -1;
  if (!shape) return r2 >= 25.0 ? 2 : -1;
  return r2 >= 625.0 && kR2 <= 0.04 ? 4 : r2 >= 64.0 && kR2 <= 0.25 ? 3 : r2 >= 25.0 ? 2 : r2 >= 12.25 ? 1 : r2 >= 9.0 ? 0 : -1;
}
// The same for a part of a pair that is not its nearest image: flat quads
// inside the shape guard reach 2e-13 of the image's largest entry with 7 points
// from 6 R and with 6 from 10 R (k R <= 0.5; numpy, random directions, twists and
// aspects inside the guard), so 7 from 7 R and 6 from 12 R here.
__device__ __forceinline__ int tier_image(double r2, double kR2, bool tri, bool shape) {
  if (tri || !shape) return tier_of(r2, kR2, tri, shape);
  if (kR2 > 1.0) return -1;
  return r2 >= 144.0 && kR2 <= 0.25 ? 4 : r2 >= 49.0 && kR2 <= 0.25 ? 3 : r2 >= 25.0 ? 2 : r2 >= 12.25 ? 1 : r2 >= 9.0 ? 0 : -1;
}
// Free space, with the tangential derivatives of G and H (a third-order
// singularity), and the geometric sums: 1e-14 of the largest entry of each
// matrix, the rounding of the 144-point sums themselves (numpy, as above; quads
// and triangles alike): 10 points from 4 R, 9 from 5, 8 from 7, 7 from 9
// (k R <= 0.5), 6 from 16 (k R <= 0.25).
__device__ __forceinline__ int tier_free(double r2, double kR2, bool shape) {
  if (kR2 > 1.0 || !shape) return -1;
  return r2 >= 256.0 && kR2 <= 0.0625 ? 4 : r2 >= 81.0 && kR2 <= 0.25 ? 3 : r2 >= 49.0 ? 2 : r2 >= 25.0 ? 1 : r2 >= 16.0 ? 0 : -1;
}
// points of rule n on an element: 12 is the reference's 12 x 12 (3 parts of it on
// a triangle), 6 .. 10 a tier's n x n; point pt of it, its weight as those of the
// 12 x 12 rules (relative to W)
__device__ __forceinline__ int rule_npts(int n, bool tri) { return n == BEM_GLN && tri ? 3 * BEM_GLN * BEM_GLN : n * n; }
__device__ __forceinline__ void tier_point(int t, bool tri, int i, int j, double &z, double &e);
__device__ __forceinline__ void rule_pt(int n, bool tri, int pt, double &z, double &e, double &wt) {
  if (n == BEM_GLN) {
    const int part = pt / (BEM_GLN * BEM_GLN), ij = pt % (BEM_GLN * BEM_GLN);
    const double a = c_q.xl[ij / BEM_GLN], c = c_q.xl[ij % BEM_GLN];
    z = a;
    e = c;
    wt = c_q.wl[ij / BEM_GLN] * c_q.wl[ij % BEM_GLN];
    if (tri) {
      bem_tri_point(part, a, c, z, e);
      wt *= bem_tri_wfac(a, c);
    }
  } else {
    const int t = BEM_TIER_N0 - n, i = pt / n, j = pt - i * n;
    tier_point(t, tri, i, j, z, e);
    wt = c_q.wt[t][i] * c_q.wt[t][j];
    if (tri) wt *= 0.125 * (c_q.xt[t][i] + 1.0);
  }
}
// point (i, j) of tier t's rule: Gauss on a quad; on a triangle the collapsed
// (Duffy) rule over the whole reference triangle, (z, e) = (1 - 3u/2,
// sqrt3/2 u (1 - 2v)) for (u, v) in [0, 1]^2, weight u w_u w_v
__device__ __forceinline__ void tier_point(int t, bool tri, int i, int j, double &z, double &e) {
  if (tri) {
    const double u = 0.5 * (c_q.xt[t][i] + 1.0), v = 0.5 * (c_q.xt[t][j] + 1.0);
    z = 1.0 - 1.5 * u;
    e = 0.5 * BEM_SQ3 * u * (1.0 - 2.0 * v);
  } else {
    z = c_q.xt[t][i];
    e = c_q.xt[t][j];
  }
}
