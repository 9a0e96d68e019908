// Source points of the field and boundary sums, the singular polar rule and the
// home image, shared by the pointwise kernels (bem_post.cuh, bem_assemble.cu) and
// those with images and expansion (bem_smooth.cu).  Needs bem_qpgf.cuh, bem_geom.cuh.
#pragma once
#include "bem_kernels.h"

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void set_status(unsigned *st, unsigned bits) { if (bits) atomicOr(st, bits); }
// Quadrature points closer than this to the lattice plane through the node
// keep a pair on the reference's rule: there the reference's lattice sums
// stop on rounding-decided zeros, so its values at its own points are not a
// smooth function that another rule could reproduce.
#define BEM_FAR_PLANE_TOL 1e-10

// ------------------------------------------------------------------ rules of the field and boundary sums
// rule point idx of a source element: parameter point, weight, node flag
__device__ __forceinline__ int rule_points(int type) {
  return type == 0 ? 4 : (type == 1 ? 9 : (type == 2 ? BEM_GLN * BEM_GLN : BEM_GHN * BEM_GHN));
}

__device__ __forceinline__ void rule_point(int type, int i, double &z, double &e, double &w) {
  if (type == 0) { z = c_q.zt[i]; e = c_q.et[i]; w = 1.0; }
  else if (type == 1) { z = c_q.z9[i]; e = c_q.e9[i]; w = c_q.w9[i]; }
  else if (type == 2) { z = c_q.xl[i / BEM_GLN]; e = c_q.xl[i % BEM_GLN]; w = c_q.wl[i / BEM_GLN] * c_q.wl[i % BEM_GLN]; }
  else { z = c_q.xh[i / BEM_GHN]; e = c_q.xh[i % BEM_GHN]; w = c_q.wh[i / BEM_GHN] * c_q.wh[i % BEM_GHN]; }
}

// Rules on a triangle source (q0_lit_coef_4p / _7p / _GL / _GH, q0_lit_coef.c:10-250):
// type 0: the 3 nodes and the centre (weights 25/48 x 3, -27/48), 1: 7-point rule,
// 2, 3: the 3-part 12 x 12 / 64 x 64 rules.  w multiplies W = cw0 (twice the area).
__device__ __forceinline__ int tri_rule_points(int type) {
  return type == 0 ? 4 : (type == 1 ? 7 : 3 * (type == 2 ? BEM_GLN * BEM_GLN : BEM_GHN * BEM_GHN));
}
__device__ __forceinline__ void tri_rule_point(int type, int i, double &z, double &e, double &w) {
  if (type == 0) {
    if (i < 3) bem_tri_node(i, z, e);
    else z = e = 0.0;
    w = 0.5 * (i < 3 ? 25.0 / 48.0 : -27.0 / 48.0);
  } else if (type == 1) {
    // the 7-point rule (zt_37, et_37, wt_37, bem3_aw_qd2.c:1012-1021)
    const double n0 = 0.3480702390148154917985, n1 = 0.2052130961576726346557;
    const double n2 = 0.6028753385763033130539, n3 = 0.3554395089236065568357;
    const double v0 = 0.1259391805448271525957, v1 = 0.1323941527885061807376, v2 = 0.225;
    const double zz[7] = {-n0, 2.0 * n0, -n0, n1, -2.0 * n1, n1, 0.0}, ee[7] = {-n2, 0.0, n2, n3, 0.0, -n3, 0.0};
    z = zz[i];
    e = ee[i];
    w = 0.5 * (i < 3 ? v0 : (i < 6 ? v1 : v2));
  } else {
    const int n = type == 2 ? BEM_GLN : BEM_GHN;
    const double *x = type == 2 ? c_q.xl : c_q.xh, *wq = type == 2 ? c_q.wl : c_q.wh;
    const int part = i / (n * n), ij = i % (n * n), a = ij / n, b = ij % n;
    bem_tri_point(part, x[a], x[b], z, e);
    w = wq[a] * wq[b] * bem_tri_wfac(x[a], x[b]);
  }
}

// boundary values of source element s interpolated at (z,e); type 0 uses the
// node value itself (the 4-point rule sits on the nodes; the triangle's centre
// point takes the mean of its 3 nodes)
__device__ __forceinline__ void interp_bv(int type, int i, double z, double e, int s, const double *P, const double *dP,
                                          const double *pv, const double *dpv, cplx &Pn, cplx &dPn, cplx pvn[3],
                                          cplx dpvn[3], bool tri = false) {
  double N[4];
  if (type == 0 && !(tri && i == 3)) {
    for (int a = 0; a < 4; ++a) N[a] = a == i ? 1.0 : 0.0;
  } else {
    bem_Nn(tri, z, e, N);
  }
  Pn = dPn = cmk(0, 0);
  for (int c = 0; c < 3; ++c) pvn[c] = dpvn[c] = cmk(0, 0);
  for (int a = 0; a < 4; ++a) {
    const size_t o = (size_t)s * 4 + a;
    Pn = cadd(Pn, cscale(cmk(P[2 * o], P[2 * o + 1]), N[a]));
    dPn = cadd(dPn, cscale(cmk(dP[2 * o], dP[2 * o + 1]), N[a]));
    for (int c = 0; c < 3; ++c) {
      pvn[c] = cadd(pvn[c], cscale(cmk(pv[2 * (3 * o + c)], pv[2 * (3 * o + c) + 1]), N[a]));
      dpvn[c] = cadd(dpvn[c], cscale(cmk(dpv[2 * (3 * o + c)], dpv[2 * (3 * o + c) + 1]), N[a]));
    }
  }
}

// point i of the rule of source element s (0-based in the domain's list, se the
// element) of a boundary sum: (z, e), weight, r, W
__device__ __forceinline__ void bd_source_point(const bem_dom_dev &D, int se, bool stri, int type, int i, double &z,
                                                double &e, double &w, double r[3], double vW[3]) {
  if (stri) tri_rule_point(type, i, z, e, w);
  else rule_point(type, i, z, e, w);
  if (type == 0 && !(stri && i == 3)) {
    for (int d = 0; d < 3; ++d) {
      r[d] = __ldg(D.ren + (size_t)se * 12 + i * 3 + d);
      vW[d] = __ldg(D.wen + (size_t)se * 12 + i * 3 + d);
    }
  } else {
    bem_el el;
    bem_load_el(D.cr, D.cw, se, el);
    bem_rw_ref(el, z, e, r, vW);
  }
}

// The geometric sum F of a field point and its gradient, times 4 pi: sw (sign and weight)
// times (R . W) / R^3 to a[0], its gradient to a[1 .. 3].  Over a closed body the sum
// cancels to 1e-8 of its terms, so every kernel that forms it rounds alike: each
// operation is spelled out.
__device__ __forceinline__ void fld_geom(const double R[3], const double W[3], double sw, double *a) {
  const double r2 = __fma_rn(R[2], R[2], __fma_rn(R[1], R[1], __dmul_rn(R[0], R[0])));
  const double iR = __ddiv_rn(1.0, __dsqrt_rn(r2));
  const double rdW = __dmul_rn(__fma_rn(R[2], W[2], __fma_rn(R[1], W[1], __dmul_rn(R[0], W[0]))), iR);
  a[0] = __fma_rn(__dmul_rn(__dmul_rn(sw, rdW), iR), iR, a[0]);
  const double s3 = __dmul_rn(sw, __dmul_rn(__dmul_rn(iR, iR), iR));
#pragma unroll
  for (int j = 0; j < 3; ++j)
    a[1 + j] = __fma_rn(s3, __fma_rn(__dmul_rn(__dmul_rn(3.0, R[j]), iR), rdW, -W[j]), a[1 + j]);
}

// ------------------------------------------------------------------ polar rule
struct polar_pt { double th, wth; int j; };
__device__ __forceinline__ polar_pt polar_theta(const double th[5], int idx /* 0..511 */) {
  const int j = idx >> 7, h = (idx >> 6) & 1, m = idx & 63;
  const double t0 = th[j], t1 = th[j + 1];
  polar_pt r;
  r.th = h == 0 ? 0.25 * (t1 - t0) * c_q.xh[m] + 0.25 * (t1 + 3.0 * t0) : 0.25 * (t1 - t0) * c_q.xh[m] + 0.25 * (3.0 * t1 + t0);
  r.wth = c_q.wh[m] * 0.25 * (t1 - t0);
  r.j = j;
  return r;
}

// The rule's angles as a table in shared memory (nang <= 512): cosine, sine,
// radius to the edge, weight.  Each angle serves 12 or 64 radii, whose points
// otherwise form its four trigonometric functions again.  All threads; the
// caller synchronises.
#define POLAR_N 512
struct polar_tab { double c[POLAR_N], s[POLAR_N], rm[POLAR_N], w[POLAR_N]; };
__device__ __forceinline__ void polar_fill(polar_tab &T, const double r[5], const double th[5], int nang, unsigned &st) {
  for (int i = threadIdx.x; i < nang; i += blockDim.x) {
    const polar_pt tp = polar_theta(th, i);
    const double rm = bem_rmax(r[tp.j], r[tp.j + 1], th[tp.j], th[tp.j + 1], tp.th);
    if (rm < 0.0) st |= BEM_ST_GEOMETRY;
    sincos(tp.th, &T.s[i], &T.c[i]);
    T.rm[i] = rm;
    T.w[i] = tp.wth;
  }
}

// geometric F of the element at parameter point (zt,et) by the polar rule (q0_bil_coef_bd_F,
// q0_bil_dcoef_v2_cc.c:401-454 / bil_sF_theta): returns the un-normalised sum (times bdC/4pi later)
static __device__ double polar_F_partial(const bem_el &el, double zt, double et, unsigned &st) {
  double r[5], th[5];
  bem_node_r_th(zt, et, r, th);
  double acc = 0.0;
  for (int idx = threadIdx.x; idx < 512; idx += blockDim.x) {
    const polar_pt tp = polar_theta(th, idx);
    const double rm = bem_rmax(r[tp.j], r[tp.j + 1], th[tp.j], th[tp.j + 1], tp.th);
    if (rm < 0.0) st |= BEM_ST_GEOMETRY;
    double sth, cth;
    sincos(tp.th, &sth, &cth);
    double inner = 0.0;
    for (int ir = 0; ir < BEM_GLN; ++ir) {
      const double rr = 0.5 * rm * (c_q.xl[ir] + 1.0);
      double K[3];
      bem_K(el, rr, cth, sth, zt, et, K);
      const double aK = sqrt(K[0] * K[0] + K[1] * K[1] + K[2] * K[2]);
      inner += c_q.wl[ir] / (aK * aK * aK) * cth * sth;
    }
    acc += tp.wth * 0.5 * rm * inner;
  }
  return acc;
}

__device__ __forceinline__ double bem_bdC(const bem_el &el) {
  return el.cr[0][1] * el.cw[0][2] + el.cr[1][1] * el.cw[1][2] + el.cr[2][1] * el.cw[2][2];
}

// The home-cell image of the quasi-periodic Green's function: the free-space
// e^{ikR} / (4 pi R) and its gradient at r, in bem_qpgf's conventions.  The
// near-singular and self integrals split G_qp = G0 + (G_qp - G0): G0 carries
// the whole singularity and costs a sincos, so it is integrated on the
// reference's own points (64 x 64 Gauss, the polar rule); the rest is smooth
// over the element (its nearest singularities are the other lattice images)
// and is integrated on the 12 x 12 Gauss rule of regular pairs, a lattice sum
// at 144 points instead of 4096 or 6144.
__device__ __forceinline__ void bem_g0(double k, const double vR[3], bem_gval &o) {
  const double R2 = vR[0] * vR[0] + vR[1] * vR[1] + vR[2] * vR[2];
  const double R = sqrt(R2), iR = 1.0 / R;
  const cplx ce = cexpi(k * R);
  const double c4 = 0.07957747154594766788 * iR;  // 1 / (4 pi R)
  o.g = cscale(ce, c4);
  // (i k R - 1) e^{ikR} / (4 pi R^3) times r
  const cplx f = cscale(cmul(cmk(-1.0, k * R), ce), c4 * iR * iR);
  o.gx = cscale(f, vR[0]);
  o.gy = cscale(f, vR[1]);
  o.gz = cscale(f, vR[2]);
}
