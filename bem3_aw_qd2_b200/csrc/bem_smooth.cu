// Regular part of the periodic domain's coefficient matrices without lattice
// sums per quadrature point.
//
// The quasi-periodic Green's function of R = y - x (source minus collocation
// point) is split into the lattice images that can come near,
//   G_qp(R) = sum_{l in I} e^{i k_par . R_l} e^{ik|R + R_l|} / (4 pi |R + R_l|) + G_s(R),
// and a rest G_s that solves the Helmholtz equation in |R| < c, c the distance
// of the nearest image left in it.  With the body inside a ball of radius R0
// about its centre, c > 2 R0, the rest is an expansion in regular waves,
//   G_s(y - x) = sum_{lm, l'm'} phi_lm(y) T_lm,l'm' phi_l'm'(x),
// which separates source and target: the integrals over the elements become
// one matrix V = [int N_a |W| phi | int N_a W . grad phi] (K x 8 ne), the
// targets one matrix A = U T, and the rest of every pair of G and H one real
// matrix product on the FP64 tensor cores.  The reference sums about 110
// lattice terms at each of the 36 to 144 points of every pair
// (q0_bil_dcoef_v2_cc.c:129-204 over d3_qpgf_d2.c:124-176); here a pair costs
// 16 K multiply-adds of the product and a closed form per image and point.
//
// The images keep the quadrature rule of their own distance (bem_tiers.cuh), so
// every part meets the accuracy of the pairwise rules; pairs with a point on
// the lattice plane through their node stay with the kernels that sum the
// lattice point by point (the reference's sums stop on rounding there).
//
// 216-quad sphere, square lattice of 0.8 wavelengths (K = 625): 1.25 ms of kernels in
// place of 17.3 ms of lattice sums at the points.  The split alone took the whole
// solve from 28.5 to 11.9 ms, of the 1536-quad sphere from 957 to 374 ms, of 320
// triangles from 70 to 29 ms.
//
// phi_lm(y) = g_l(k r) R_lm((y - centre) / R0), g_l(z) = (2l + 1)!! j_l(z) / z^l
// (entire, near 1), R_lm real orthonormal solid harmonics: no zeros of j_l, no
// large or small factors.  The coefficients of G_s come from its values and
// radial derivatives on the sphere |R| = 2 R0 (Ewald sums at about 3000 points),
// projected on spherical harmonics; T from them by the addition theorem, its
// Gaunt integrals by Gauss-Legendre quadrature (exact for these degrees).
#include "bem_count.h"
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <algorithm>
#include <vector>
#include "bem_qpgf.cuh"
#include "bem_geom.cuh"
#include "bem_tiers.cuh"
#include "bem_kernels.h"
#include "bem_rules.cuh"
#include "bem_smooth.h"


// ------------------------------------------------------------------ host: the split
// |j_l(z)| = z^l g_l / (2l + 1)!! and |h_l(z)| for l = 0 .. n
static void bessel_sizes(int n, double z, std::vector<double> &j, std::vector<double> *h) {
  const int top = n + 20 + (int)z;
  std::vector<double> g(top + 2);
  for (int l = top; l <= top + 1; ++l) {
    double t = 1.0, s = 1.0;
    for (int m = 1; m < 200 && fabs(t) > 1e-20 * fabs(s); ++m) {
      t *= -0.5 * z * z / (m * (2.0 * l + 2.0 * m + 1.0));
      s += t;
    }
    g[l] = s;
  }
  for (int l = top; l > 0; --l) g[l - 1] = g[l] - z * z / ((2.0 * l + 1.0) * (2.0 * l + 3.0)) * g[l + 1];
  j.assign(n + 1, 0.0);
  double f = 1.0;
  for (int l = 0; l <= n; ++l) {
    j[l] = f * g[l];
    f *= z / (2.0 * l + 3.0);
  }
  if (!h) return;
  h->assign(n + 1, 0.0);
  double y0 = -cos(z) / z, y1 = -cos(z) / (z * z) - sin(z) / z;
  for (int l = 0; l <= n; ++l) {
    (*h)[l] = sqrt(j[l] * j[l] + y0 * y0);
    const double y2 = (2.0 * l + 3.0) / z * y1 - y0;
    y0 = y1;
    y1 = y2;
  }
}
// smallest degree whose terms k (2l + 1) |j_l(k a) h_l(k b)| beyond it stay
// below tol / scale; -1: none up to lim
static int degree_for(double k, double a, double b, double scale, double tol, int lim) {
  std::vector<double> j, h;
  bessel_sizes(lim + 4, k * a, j, nullptr);
  std::vector<double> jb;
  bessel_sizes(lim + 4, k * b, jb, &h);
  for (int l = lim; l >= 0; --l) {
    const double e = k * (2.0 * (l + 1) + 1.0) * fabs(j[l + 1]) * h[l + 1] * scale;
    if (!(e <= tol)) return l == lim ? -1 : l + 1;
  }
  return 0;
}

// The BEM_SM_MAXIMG + 1 lattice points nearest to the origin, by distance (those of one
// distance in order of their indices).  S->np = 0 where the lattice's basis is too
// skewed, or the body too many periods wide, for a split to be looked for.
static void nearest_points(bem_smooth *S, const bem_qp *q) {
  struct pt { double r; int a, b; };
  S->np = 0;
  const double g1 = hypot(q->g1x, q->g1y) / (2.0 * M_PI), g2 = hypot(q->g2x, q->g2y) / (2.0 * M_PI);
  const double wide = 12.0 * S->R0 + 4.0 * (hypot(q->d1x, q->d1y) + hypot(q->d2x, q->d2y));
  if (!((floor(wide * g1) + 1) * (floor(wide * g2) + 1) <= 1e5)) return;
  std::vector<pt> P;
  const size_t want = BEM_SM_MAXIMG + 1;
  // every point within the reach is listed; a disc of the wanted points' area holds
  // about as many, a wider one more
  for (double reach = 1.2 * sqrt(want / (M_PI * q->aidet)); P.size() < want; reach *= 1.4) {
    P.clear();
    const int n1 = (int)floor(reach * g1) + 1, n2 = (int)floor(reach * g2) + 1;
    for (int a = -n1; a <= n1; ++a)
      for (int b = -n2; b <= n2; ++b) {
        const double r = hypot(a * q->d1x + b * q->d2x, a * q->d1y + b * q->d2y);
        if (r <= reach) P.push_back({r, a, b});
      }
  }
  std::stable_sort(P.begin(), P.end(), [](const pt &x, const pt &y) { return x.r < y.r; });
  S->np = (int)want;
  for (size_t i = 0; i < want; ++i) {
    S->pr[i] = P[i].r;
    S->p1[i] = P[i].a;
    S->p2[i] = P[i].b;
  }
}
static void finish_plan(bem_smooth *S, const bem_qp *q);
static void take_images(bem_smooth *S) {
  S->cut = S->pr[S->nimg] - S->rho;
  for (int i = 0; i < S->nimg; ++i) {
    S->l1[i] = S->p1[i];
    S->l2[i] = S->p2[i];
  }
}

void bem_smooth_plan(bem_smooth *S, const bem_qp *q, const double *cr, const int *npe, const int *sid, int ne) {
  S->on = 0;
  S->have0 = S->have1 = 0;
  if (ne <= 0) return;
  // the ball of the body: corners (+-1, +-1) of a quad, (1, 0), (-1/2,
  // +-sqrt3/2) of a triangle; every point of an element is a convex
  // combination of its corners
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  auto corners = [&](int s, double (*v)[3]) {
    const int e = abs(sid[s]) - 1, n = npe[e] == 3 ? 3 : 4;
    const double zq[4] = {-1, 1, 1, -1}, eq[4] = {-1, -1, 1, 1};
    const double zt[3] = {1.0, -0.5, -0.5}, et[3] = {0.0, 0.86602540378443864676, -0.86602540378443864676};
    for (int c = 0; c < n; ++c) {
      const double z = n == 3 ? zt[c] : zq[c], w = n == 3 ? et[c] : eq[c];
      for (int d = 0; d < 3; ++d) {
        const double *r = cr + (size_t)e * 12 + 4 * d;
        v[c][d] = r[0] + r[1] * z + r[2] * w + r[3] * z * w;
      }
    }
    return n;
  };
  double v[4][3];
  for (int s = 0; s < ne; ++s) {
    const int n = corners(s, v);
    for (int c = 0; c < n; ++c)
      for (int d = 0; d < 3; ++d) { lo[d] = std::min(lo[d], v[c][d]); hi[d] = std::max(hi[d], v[c][d]); }
  }
  for (int d = 0; d < 3; ++d) S->ctr[d] = 0.5 * (lo[d] + hi[d]);
  double R2 = 0.0;
  for (int s = 0; s < ne; ++s) {
    const int n = corners(s, v);
    for (int c = 0; c < n; ++c) {
      double r2 = 0.0;
      for (int d = 0; d < 3; ++d) r2 += (v[c][d] - S->ctr[d]) * (v[c][d] - S->ctr[d]);
      R2 = std::max(R2, r2);
    }
  }
  S->R0 = sqrt(R2) * (1.0 + 1e-12);
  S->rho = 2.0 * S->R0;
  S->k = q->k;
  if (!(S->R0 > 0.0) || !std::isfinite(S->R0)) return;
  nearest_points(S, q);
  // the cheapest split, in FP64 operations at the rates that the kernels reach
  // (images 0.55 of the pipe, the product 0.7): per pair about 45 points of 66
  // for each image and 16 multiply-adds for each of the K functions (G and H of
  // 4 entries, complex); once, A = U T, the samples (about 300 terms of 100 each)
  // and T.  Summed point by point a pair takes about 8e5 at half the pipe.
  const double pairs = 4.0 * ne * ne;
  double best = 1e6 * pairs;
  for (int c = S->np - 1; c >= 1; --c) {
    if (S->pr[c] <= S->pr[c - 1] * (1.0 + 1e-9)) continue;  // whole shells only
    const double cut = S->pr[c], images = pairs * (c - 1) * 45.0 * 66.0 / 0.55;
    if (cut <= S->rho * 1.05) break;
    if (images >= best) continue;
    // tail relative to 1 / (4 pi 2 R0), six images on the first shell left in
    const int lmax = degree_for(S->k, S->R0, cut - S->R0, 6.0 * S->rho, 1e-15, BEM_SM_MAXL);
    if (lmax < 0) continue;
    int Lmax = degree_for(S->k, S->rho, cut, 6.0 * S->rho, 1e-15, 2 * BEM_SM_MAXL);
    if (Lmax < 0 || Lmax > 2 * lmax) Lmax = 2 * lmax;
    const double K = (lmax + 1.0) * (lmax + 1.0), nt = lmax + 0.5 * Lmax + 1.0;
    const double cost = images + pairs * 16.0 * K / 0.7 + 4.0 * ne * 2.0 * K * K / 0.7 +
                        nt * (2.0 * Lmax + 2.0) * 3e4 + 0.25 * K * K * lmax * nt;
    if (cost < best) {
      best = cost;
      S->on = 1;
      S->lmax = lmax;
      S->Lmax = Lmax;
      S->nimg = c;
    }
  }
  if (!S->on) return;
  take_images(S);
  // degrees for one point's rest at |R| <= (i + 1) 2 R0 / 8 (the gradient's terms are
  // those of the value times l / |R|)
  for (int i = 0; i < 8; ++i) {
    const double f = (i + 1) / 8.0;
    const int l = degree_for(S->k, f * S->rho, S->cut + S->rho, 6.0 * S->rho, f * 1e-15, S->Lmax);
    S->lcut[i] = l < 0 ? S->Lmax : l;
  }
  finish_plan(S, q);
}

// The split for sums at points up to Rx from the body's centre: the larger ball
// takes R0's place, the degrees follow from both (a source at R0 against images
// seen from Rx, a point at Rx against images seen from R0).
double bem_smooth_plan_field(bem_smooth *F, const bem_smooth *S, const bem_qp *q, double Rx, double n, double sources,
                             double limit) {
  F->on = 0;
  F->have0 = F->have1 = 0;
  F->inst = 1;
  F->first = 0;
  F->k = q->k;
  for (int d = 0; d < 3; ++d) F->ctr[d] = S->ctr[d];
  F->R0 = std::max(Rx, S->R0) * (1.0 + 1e-12);
  F->rho = F->R0 + S->R0;
  double best = limit;
  if (!(F->R0 < 1e3 * S->R0)) return 1e300;
  F->np = S->np;
  std::copy(S->pr, S->pr + S->np, F->pr);
  std::copy(S->p1, S->p1 + S->np, F->p1);
  std::copy(S->p2, S->p2 + S->np, F->p2);
  for (int c = F->np - 1; c >= 1; --c) {  // as bem_smooth_plan
    if (F->pr[c] <= F->pr[c - 1] * (1.0 + 1e-9)) continue;
    // an image with second derivatives about 160 operations, a pair's own part 400
    const double cut = F->pr[c], images = n * sources * (400.0 + c * 160.0) / 0.55;
    if (cut <= F->rho * 1.05) break;
    if (images >= best) continue;
    const int lx = degree_for(F->k, F->R0, cut - S->R0, 6.0 * F->rho, 1e-15, BEM_SM_MAXL);
    if (lx < 0) continue;
    const int ly = degree_for(F->k, S->R0, cut - F->R0, 6.0 * F->rho, 1e-15, BEM_SM_MAXL);
    if (ly < 0) continue;
    const int lmax = std::max(lx, ly);
    int Lmax = degree_for(F->k, F->rho, cut, 6.0 * F->rho, 1e-15, 2 * BEM_SM_MAXL);
    if (Lmax < 0 || Lmax > 2 * lmax) Lmax = 2 * lmax;
    const double K = (lmax + 1.0) * (lmax + 1.0), nt = lmax + 0.5 * Lmax + 1.0;
    const double cost = images + nt * (2.0 * Lmax + 2.0) * 3e4 + 0.25 * K * K * lmax * nt + sources * K * 60.0;
    if (cost < best) {
      best = cost;
      F->on = 1;
      F->lmax = lmax;
      F->Lmax = Lmax;
      F->nimg = c;
    }
  }
  if (!F->on) return 1e300;
  take_images(F);
  finish_plan(F, q);
  return F->on ? best : 1e300;
}

static void finish_plan(bem_smooth *S, const bem_qp *q) {
  // windows of the samples' Ewald sums: the reference's parameter below its cap
  // (k^2 eta^2 < 3); terms to e^{-40} of the leading one; the images among them
  S->eta = std::min(q->eta0, 0.98 * sqrt(3.0) / S->k);
  const double cutr = S->rho + 2.0 * S->eta * sqrt(40.0 + S->k * S->k * S->eta * S->eta);
  const double cuts = sqrt(40.0 / (S->eta * S->eta) + S->k * S->k);
  const double tp = 2.0 * M_PI;
  S->r1 = (int)(cutr * hypot(q->g1x, q->g1y) / tp) + 1;
  S->r2 = (int)(cutr * hypot(q->g2x, q->g2y) / tp) + 1;
  for (int i = 0; i < S->nimg; ++i) {
    S->r1 = std::max(S->r1, abs(S->l1[i]));
    S->r2 = std::max(S->r2, abs(S->l2[i]));
  }
  // a_n = -k_par + n g: |n1 - k_par . d1 / 2 pi| <= |a| |d1| / 2 pi, and for n2
  S->s1 = (int)(cuts * hypot(q->d1x, q->d1y) / tp) + 2;
  S->s2 = (int)(cuts * hypot(q->d2x, q->d2y) / tp) + 2;
  // a batch's instances share the window: centred on n2 = 0, wide enough for |k_par| <= k
  S->s2 += (int)(S->k * hypot(q->d2x, q->d2y) / tp) + 1;
  if ((double)(2 * S->r1 + 1) * (2 * S->r2 + 1) > 20000.0 || (double)(2 * S->s1 + 1) * (2 * S->s2 + 1) > 20000.0) {
    S->on = 0;
    return;
  }
  S->K = (S->lmax + 1) * (S->lmax + 1);
  S->Kp = (S->K + 15) / 16 * 16;
  // Gauss-Legendre nodes in cos(theta): exact for products of three harmonics
  // (degree 2 lmax + Lmax), an even number (no node on the lattice plane)
  S->nt = (2 * S->lmax + S->Lmax) / 2 + 1;
  S->nt += S->nt & 1;
  S->nphi = 2 * S->Lmax + 2;
}

bem_smooth_tab bem_smooth_layout(const bem_smooth *S) {
  bem_smooth_tab t;
  int o = 0;
  auto put = [&o](int n) { const int p = o; o += n; return p; };
  t.x = put(S->nt);
  t.w = put(S->nt);
  t.ca = put(S->Lmax + 1);
  t.cb = put(S->Lmax + 1);
  t.dL = put(S->Lmax + 1);
  t.el = put(S->lmax + 1);
  t.rec = put((S->Lmax + 1) * (S->Lmax + 2));
  t.img = put(3 * S->nimg * S->inst);
  t.total = o;
  return t;
}

void bem_smooth_tables(const bem_smooth *S, const bem_qp *qps, double *h) {
  const bem_smooth_tab t = bem_smooth_layout(S);
  const int n = S->nt, L = S->Lmax;
  // Gauss-Legendre by Newton's method on P_n
  for (int i = 0; i < n / 2; ++i) {
    double z = cos(M_PI * (i + 0.75) / (n + 0.5)), dp = 1.0;
    for (int it = 0; it < 60; ++it) {
      double p0 = 1.0, p1 = z;
      for (int m = 2; m <= n; ++m) {
        const double p2 = ((2.0 * m - 1.0) * z * p1 - (m - 1.0) * p0) / m;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (z * p1 - p0) / (z * z - 1.0);
      const double dz = p1 / dp;
      z -= dz;
      if (fabs(dz) < 1e-16) break;
    }
    h[t.x + i] = z;
    h[t.x + n - 1 - i] = -z;
    h[t.w + i] = h[t.w + n - 1 - i] = 2.0 / ((1.0 - z * z) * dp * dp);
  }
  // u_LM and rho u'_LM / (L + 1) are sigma_LM times g_L(k rho) and
  // (L g_L - z^2 g_{L+1} / (2L + 3)) / (L + 1): both used, no zero shared
  std::vector<double> j;
  const double z = S->k * S->rho;
  bessel_sizes(L + 1, z, j, nullptr);
  std::vector<double> g(L + 2);
  double f = 1.0;
  for (int l = 0; l <= L + 1; ++l) {
    g[l] = j[l] / f;
    f *= z / (2.0 * l + 3.0);
  }
  const double kR0 = S->k * S->R0;
  double dl = 1.0, el = 1.0;
  for (int l = 0; l <= L; ++l) {
    const double a = g[l], b = (l * g[l] - z * z / (2.0 * l + 3.0) * g[l + 1]) / (l + 1.0), s = 1.0 / (a * a + b * b);
    h[t.ca + l] = a * s;
    h[t.cb + l] = b * s / (l + 1.0);
    // (2L + 1)!! / (k rho)^L and (k R0)^l / (2l + 1)!!: j_l in terms of g_l and R_lm
    h[t.dL + l] = dl;
    dl *= (2.0 * l + 3.0) / z;
    if (l <= S->lmax) h[t.el + l] = el;
    el *= kR0 / (2.0 * l + 3.0);
  }
  // Theta_lm = a (z Theta_{l-1,m} - b s Theta_{l-2,m}), and Theta_mm at l = m
  double mm = 0.28209479177387814347;  // 1 / sqrt(4 pi)
  for (int m = 0; m <= L; ++m) {
    for (int l = m; l <= L; ++l) {
      double *r = h + t.rec + l * (l + 1) + 2 * m;
      if (l == m) {
        r[0] = mm;
        r[1] = 0.0;
      } else {
        r[0] = sqrt((4.0 * l * l - 1.0) / ((double)l * l - (double)m * m));
        r[1] = sqrt(((l - 1.0) * (l - 1.0) - (double)m * m) / (4.0 * (l - 1.0) * (l - 1.0) - 1.0));
      }
    }
    mm *= sqrt((2.0 * m + 3.0) / (2.0 * m + 2.0));
  }
  for (int b = 0; b < S->inst; ++b)
    for (int i = 0; i < S->nimg; ++i) {
      const bem_qp &q = qps[b];
      const double sx = S->l1[i] * q.d1x + S->l2[i] * q.d2x, sy = S->l1[i] * q.d1y + S->l2[i] * q.d2y;
      double *m = h + t.img + 3 * (b * S->nimg + i);
      m[0] = sx;
      m[1] = sy;
      m[2] = (q.kx * sx + q.ky * sy) * 0.31830988618379067154;  // phase / pi
    }
}

// ------------------------------------------------------------------ device view
struct sm_dev {
  int lmax, Lmax, Mx, K, Kp, nt, nphi, nimg, nlm;  // nlm: pairs (l, m >= 0) up to Lmax
  double cx, cy, cz, R0, iR0, kR0, rho, k, cut;
  double eta;                       // Ewald parameter of the samples
  int nreal, r1, r2, nspec, s1, s2;  // its windows: l1 in [-r1, r1], l2 in [-r2, r2]; n1 - nc1 in [-s1, s1], n2 in [-s2, s2]
  int iml[2 * BEM_SM_MAXIMG];       // the images' indices
  int lcut[8];                      // degrees of the expansion about a point at |R| <= (i + 1) 2 R0 / 8
  const double *x, *w, *ca, *cb, *dL, *el, *rec, *img;
  double *plm;            // [nt][lm >= 0] normalised Legendre functions P_lm(x_t)
  double *samp;           // [nb][2][nt][nphi] complex: G_s and rho dG_s/drho
  double *sig;            // [nb][(Lmax + 1)^2] complex
  double *F;              // [nb][Lmax + 1][nt / 2][2 Mx + 1] complex: partial sums over L (k_sm_F)
  double *T;              // [nb][Kp][2 Kp]: T^t, real and imaginary parts
  double *Z, *Zt;         // densities of boundary sums: [32][Kp][8], [Kp][8]
  double *U, *V, *A;      // [4 ne][Kp], [Kp][8 ne], [nb][4 ne][2 Kp]
};
// What stays valid after an assembly (for boundary sums): Legendre functions,
// samples, sigma, T of up to BEM_SM_BAT instances, the densities
struct sm_keep { size_t plm, samp, sig, F, T, Z, Zt, total; };
static sm_keep keep_layout(const bem_smooth *S) {
  sm_keep w;
  size_t o = 0;
  auto put = [&o](size_t n) { const size_t p = o; o += (n + 31) / 32 * 32; return p; };
  const size_t L = S->Lmax, Kp = S->Kp, nb = std::min(S->inst, BEM_SM_BAT);
  w.plm = put((L + 1) * (L + 2) / 2 * S->nt);
  w.samp = put(nb * 4 * S->nt * S->nphi);
  w.sig = put(nb * 2 * (L + 1) * (L + 1));
  w.F = put(nb * 2 * (L + 1) * (S->nt / 2) * (2 * std::min(2 * S->lmax, S->Lmax) + 1));
  w.T = put(nb * 2 * Kp * Kp);
  w.Z = put(32 * Kp * 8);
  w.Zt = put((Kp + 1) * 8);
  w.total = o;
  return w;
}
size_t bem_smooth_keep_doubles(const bem_smooth *S) { return keep_layout(S).total; }
// and an assembly's scratch
struct sm_ws { size_t U, V, A, total; };
static sm_ws ws_layout(const bem_smooth *S, int ne) {
  sm_ws w;
  size_t o = 0;
  auto put = [&o](size_t n) { const size_t p = o; o += (n + 31) / 32 * 32; return p; };
  const size_t Kp = S->Kp, nb = std::min(S->inst, BEM_SM_BAT);
  w.U = put(4 * (size_t)ne * Kp);
  w.V = put(8 * (size_t)ne * Kp);
  w.A = put(nb * 8 * ne * Kp);
  w.total = o;
  return w;
}
size_t bem_smooth_ws_doubles(const bem_smooth *S, int ne) { return ws_layout(S, ne).total; }

bem_smooth_room bem_smooth_need(const bem_smooth *S, int ne, size_t lent) {
  if (!S->on) return {0, 0, 0};
  const size_t tab = bem_smooth_layout(S).total, ws = bem_smooth_ws_doubles(S, ne);
  return {(tab + 31) / 32 * 32, (bem_smooth_keep_doubles(S) + 31) / 32 * 32, S->inst == 1 && ws <= lent ? 0 : ws};
}

struct sm_qps { bem_qp q[BEM_SM_BAT]; };
struct sm_out { double *G[BEM_SM_BAT], *H[BEM_SM_BAT]; };

// the closed form of one image at P = R + R_l, times e^{i pi ph}: value g and
// the factor f of its gradient f P
__device__ __forceinline__ void sm_image(double kpi, double k, double px, double py, double pz2, double ph, double &gr,
                                         double &gi, double &fr, double &fi) {
  const double r2 = fma(px, px, fma(py, py, pz2));
  const double ir = rsqrt(r2), r = r2 * ir;
  double s, c;
  sincospi(fma(kpi, r, ph), &s, &c);
  gr = ir * c;
  gi = ir * s;
  const double ir2 = ir * ir, kr = k * r;
  fr = -ir2 * fma(kr, gi, gr);
  fi = ir2 * fma(kr, gr, -gi);
}

// ------------------------------------------------------------------ coefficients of the rest
// Warps below nsamp blocks: G_s and its radial derivative at the sphere points.
// A warp takes a point, its lanes the terms of an Ewald sum over fixed windows:
// lattice points within |P| < 2 eta sqrt(40 + k^2 eta^2) of a point of the ball
// |R| <= 2 R0, orders with |beta| eta < sqrt(40 + ...): every term above 1e-17
// of the leading one, with no stopping tests, which a chain of dependent terms
// would wait for (220 us with a thread per point and the adaptive sums of
// bem_qpgf, 65 us like this).  eta keeps k eta below the reference's cap sqrt(3), so that
// e^{k^2 eta^2} costs no digits.  The other blocks: P_lm at the nodes.
#define SMP_TH 128
__global__ void __launch_bounds__(SMP_TH) k_sm_sample(const __grid_constant__ sm_dev S, const __grid_constant__ sm_qps Q,
                                                      int nsamp, unsigned *status) {
  if ((int)blockIdx.x < nsamp) {
    const int b = blockIdx.y, lane = threadIdx.x & 31, i = blockIdx.x * (SMP_TH / 32) + (threadIdx.x >> 5);
    if (i >= S.nt * S.nphi) return;
    const bem_qp &q = Q.q[b];
    const int t = i / S.nphi, jp = i % S.nphi;
    const double ct = S.x[t], sn = sqrt((1.0 - ct) * (1.0 + ct));
    double sp, cp;
    sincospi(2.0 * jp / S.nphi, &sp, &cp);
    const double ux = sn * cp, uy = sn * sp, X = S.rho * ux, Y = S.rho * uy, Z = S.rho * ct;
    const double ve = S.eta, ke = q.k * ve, kpi = S.k * 0.31830988618379067154;
    double ur = 0, ui = 0, xr = 0, xi = 0;
    // real-space terms less the images taken out, times 4 pi
    for (int e = lane; e < S.nreal; e += 32) {
      const int l1 = e / (2 * S.r2 + 1) - S.r1, l2 = e % (2 * S.r2 + 1) - S.r2;
      const double sx = l1 * q.d1x + l2 * q.d2x, sy = l1 * q.d1y + l2 * q.d2y;
      const double px = X + sx, py = Y + sy, r2 = px * px + py * py + Z * Z;
      bool out = false;  // one of the images: its closed form is not part of G_s
      for (int m = 0; m < S.nimg; ++m) out |= S.iml[2 * m] == l1 && S.iml[2 * m + 1] == l2;
      const double arg = ke * ke - r2 / (4.0 * ve * ve);
      if (arg < -42.0 && !out) continue;
      const double ph = (q.kx * sx + q.ky * sy) * 0.31830988618379067154, d = px * ux + py * uy + Z * ct;
      double s, c;
      sincospi(ph, &s, &c);
      double a = 0.0, f = 0.0;
      const double ir = rsqrt(r2), r = r2 * ir;
      if (arg >= -42.0) {
        const cplx w = bem_faddeeva(ke, r / (2.0 * ve));
        const double ef = exp(arg);
        a = ir * ef * w.re;
        f = -ir * ir * ef * (ir * w.re - q.k * w.im + 0.56418958354775628695 / ve);
      }
      ur += c * a;
      ui += s * a;
      xr += c * f * d;
      xi += s * f * d;
      if (out) {
        double gr, gi, fr, fi;
        sm_image(kpi, S.k, px, py, Z * Z, ph, gr, gi, fr, fi);
        ur -= gr;
        ui -= gi;
        xr -= fr * d;
        xi -= fi * d;
      }
    }
    ur *= BEM_I_FP; ui *= BEM_I_FP; xr *= BEM_I_FP; xi *= BEM_I_FP;
    // spectral terms (ew_spec_term)
    const double c2 = 0.25 * q.aidet, dz = Z / (2.0 * ve);
    bool ray = false;
    for (int e = lane; e < S.nspec; e += 32) {
      const int n1 = q.nc1 + e / (2 * S.s2 + 1) - S.s1, n2 = e % (2 * S.s2 + 1) - S.s2;
      const double ax = bem_an(-q.kx, n1, q.g1x, n2, q.g2x), ay = bem_an(-q.ky, n1, q.g1y, n2, q.g2y);
      const double bn2 = __dadd_rn(__dadd_rn(__dmul_rn(q.k, q.k), -__dmul_rn(ax, ax)), -__dmul_rn(ay, ay));
      if (bn2 * ve * ve < -42.0) continue;
      double s, c;
      sincos(ax * X + ay * Y, &s, &c);
      const double da = ax * ux + ay * uy;
      cplx F, D;  // sum of F_n and its z-derivative factor, before the phase
      if (bn2 > 0.0) {
        const double bn = sqrt(bn2), ef = exp(bn2 * ve * ve - dz * dz);
        const cplx ff = cexpi(bn * Z), w = bem_faddeeva(bn * ve, dz);
        F = cmk(2.0 * ff.re / bn, 2.0 * (ef * w.im + ff.im) / bn);
        D = cmk(2.0 * (ef * w.re - ff.re), -2.0 * ff.im);
      } else if (bn2 < 0.0) {
        const double bn = sqrt(-bn2), bv = bn * ve, eq = exp(-(bv * bv + dz * dz));
        const double f1 = eq * erfcx(bv + dz), f2 = eq * erfcx(bv - dz);
        F = cmk(0.0, -(f1 + f2) / bn);
        D = cmk(f1 - f2, 0.0);
      } else {
        ray = true;
        continue;
      }
      const cplx ce = cmk(c, s), Fn = cmul(ce, F), Dn = cmul(ce, D);
      // value i c2 F, gradient (-c2 a F, c2 D)
      ur -= c2 * Fn.im;
      ui += c2 * Fn.re;
      xr += c2 * (Dn.re * ct - da * Fn.re);
      xi += c2 * (Dn.im * ct - da * Fn.im);
    }
    if (ray) atomicOr(status, BEM_ST_RAYLEIGH);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ur += __shfl_down_sync(0xffffffffu, ur, o);
      ui += __shfl_down_sync(0xffffffffu, ui, o);
      xr += __shfl_down_sync(0xffffffffu, xr, o);
      xi += __shfl_down_sync(0xffffffffu, xi, o);
    }
    if (lane == 0) {
      double2 *o = reinterpret_cast<double2 *>(S.samp) + (size_t)b * 2 * S.nt * S.nphi + i;
      o[0] = make_double2(ur, ui);
      o[(size_t)S.nt * S.nphi] = make_double2(S.rho * xr, S.rho * xi);
    }
    return;
  }
  if (blockIdx.y) return;
  // P_lm(x_t): one thread per (m, t), upward in l
  const int i = (blockIdx.x - nsamp) * SMP_TH + threadIdx.x;
  if (i >= (S.Lmax + 1) * S.nt) return;
  const int m = i % (S.Lmax + 1), t = i / (S.Lmax + 1);
  const double ct = S.x[t], sn = sqrt((1.0 - ct) * (1.0 + ct));
  double p1 = S.rec[m * (m + 1) + 2 * m], p0 = 0.0;
  for (int a = 0; a < m; ++a) p1 *= sn;
  for (int l = m; l <= S.Lmax; ++l) {
    if (l > m) {
      const double *r = S.rec + l * (l + 1) + 2 * m;
      const double p2 = r[0] * (ct * p1 - r[1] * p0);
      p0 = p1;
      p1 = p2;
    }
    S.plm[(size_t)t * S.nlm + l * (l + 1) / 2 + m] = p1;
  }
}

// sigma_LM of one order M and instance: Fourier sums in phi at every node,
// then Legendre sums
#define SMC_TH 128
#define SM_MAXNT (3 * BEM_SM_MAXL + 4)
#define SMC_NJ ((4 * BEM_SM_MAXL + 2 + 31) / 32)
__global__ void __launch_bounds__(SMC_TH) k_sm_coef(const __grid_constant__ sm_dev S) {
  __shared__ double F[4][SM_MAXNT];
  const int M = (int)blockIdx.x - S.Lmax, b = blockIdx.y;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double2 *u = reinterpret_cast<const double2 *>(S.samp) + (size_t)b * 2 * S.nt * S.nphi;
  const double2 *du = u + (size_t)S.nt * S.nphi;
  // a lane's phases, the same at every node (nphi <= 4 BEM_SM_MAXL + 2 angles, 32 apart)
  double cs[SMC_NJ], sn[SMC_NJ];
#pragma unroll
  for (int i = 0; i < SMC_NJ; ++i) {
    const int j = lane + 32 * i;
    cs[i] = sn[i] = 0.0;
    if (j < S.nphi) sincospi(-2.0 * ((M * j) % S.nphi) / S.nphi, &sn[i], &cs[i]);
  }
  for (int t = wid; t < S.nt; t += SMC_TH / 32) {
    double a[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < SMC_NJ; ++i) {
      const int j = lane + 32 * i;
      if (j >= S.nphi) break;
      const double s = sn[i], c = cs[i];
      const double2 x = u[(size_t)t * S.nphi + j], y = du[(size_t)t * S.nphi + j];
      a[0] += x.x * c - x.y * s;
      a[1] += x.x * s + x.y * c;
      a[2] += y.x * c - y.y * s;
      a[3] += y.x * s + y.y * c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < 4; ++c) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
    if (lane == 0) {
      const double f = S.w[t] * 2.0 * CUDART_PI / S.nphi;
      for (int c = 0; c < 4; ++c) F[c][t] = a[c] * f;
    }
  }
  __syncthreads();
  const int am = abs(M);
  for (int l = am + threadIdx.x; l <= S.Lmax; l += SMC_TH) {
    const double *p = S.plm + l * (l + 1) / 2 + am;
    double a[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int t = 0; t < S.nt; ++t)
#pragma unroll
      for (int c = 0; c < 4; ++c) a[c] += p[(size_t)t * S.nlm] * F[c][t];
    double *o = S.sig + 2 * ((size_t)b * (S.Lmax + 1) * (S.Lmax + 1) + l * l + l + M);
    o[0] = S.ca[l] * a[0] + S.cb[l] * a[2];
    o[1] = S.ca[l] * a[1] + S.cb[l] * a[3];
  }
}

// position of the real function (l, m): cosine (or m = 0) and sine
__device__ __forceinline__ int sm_idx(int l, int m, int sine) { return l * l + (m ? 2 * m - 1 + sine : 0); }

// the real functions' entries of T from those of e^{+-i m phi}, e^{+-i m' phi}
__device__ __forceinline__ void sm_put_T(const sm_dev &S, int b, int l, int m, int l2, int m2, const cplx tp[4], double sc) {
  double *T = S.T + (size_t)b * 2 * S.Kp * S.Kp;
  auto put = [&](int r, int c, cplx z) {  // entry (source function r, target function c)
    T[(size_t)c * 2 * S.Kp + r] = sc * z.re;
    T[(size_t)c * 2 * S.Kp + S.Kp + r] = sc * z.im;
  };
  const int rc = sm_idx(l, m, 0), rs = rc + 1, cc = sm_idx(l2, m2, 0), cs = cc + 1;
  const double h2 = 0.70710678118654752440;
  if (m == 0 && m2 == 0) {
    put(rc, cc, tp[0]);
  } else if (m == 0) {
    // phi*_{+-m'} = (c -+ i s) / sqrt2: T_{0,m'}, T_{0,-m'} (tp[0], tp[1])
    put(rc, cc, cscale(cadd(tp[0], tp[1]), h2));
    put(rc, cs, cscale(cmuli(csub(tp[1], tp[0])), h2));
  } else if (m2 == 0) {
    put(rc, cc, cscale(cadd(tp[0], tp[1]), h2));
    put(rs, cc, cscale(cmuli(csub(tp[0], tp[1])), h2));
  } else {
    const cplx a = tp[0], d = tp[1], e = tp[2], g = tp[3];  // ++, --, +-, -+
    put(rc, cc, cscale(cadd(cadd(a, d), cadd(e, g)), 0.5));
    put(rs, cs, cscale(csub(cadd(a, d), cadd(e, g)), 0.5));
    // c, s': -i s' over the sign of m'; s, c': +i s over the sign of m
    put(rc, cs, cscale(cmuli(csub(cadd(d, e), cadd(a, g))), 0.5));
    put(rs, cc, cscale(cmuli(csub(cadd(a, e), cadd(d, g))), 0.5));
  }
}

// T_lm,l'm' = 4 pi sum_L sigma_{L,m-m'} i^{l-l'-L} C (2L+1)!! ... with
// C = int Y*_lm Y_l'm' Y_{L,m-m'} = 2 pi int P_lm P_l'm' P_L|m-m'| d(cos theta)
// (harmonics without the Condon-Shortley sign, Y_{l,-m} = conj Y_lm), in the
// real basis.  The sum over L goes under the integral: with
// F_M^j(t) = sum of i^-L sigma_LM ... P_L|M|(t) over L <= j, L of j's parity, an entry is
// one integral of P_lm P_l'm' F_{m-m'}^{l+l'} (L beyond l + l' integrate to zero, but
// their size would drown the rest; those below |l - l'| only round).  An integral
// for each L in its place was 16 (lmax 16) to 40 times the multiply-adds: 91 us
// for 24 quads in a period of 0.8 and 600 us for the field points' ball; with F
// 20 + 15 us and 100.
//
// F: [j <= Lmax][t][M = -Mx .. Mx], a thread per (t, M), its terms in order of L.
#define SMF_FTH 128
__global__ void __launch_bounds__(SMF_FTH) k_sm_F(const __grid_constant__ sm_dev S) {
  const int b = blockIdx.y, nM = 2 * S.Mx + 1, nh = S.nt / 2;
  const int i = blockIdx.x * SMF_FTH + threadIdx.x;
  if (i >= nM * nh) return;
  const int t = i / nM, M = i % nM - S.Mx, aM = abs(M);
  const double2 *sg = reinterpret_cast<const double2 *>(S.sig) + (size_t)b * (S.Lmax + 1) * (S.Lmax + 1);
  const double *p = S.plm + (size_t)t * S.nlm + aM;
  double2 *F = reinterpret_cast<double2 *>(S.F) + (size_t)b * (S.Lmax + 1) * nh * nM + i;
  double2 acc[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  for (int L = 0; L < aM && L <= S.Lmax; ++L) F[(size_t)L * nh * nM] = acc[0];
  // (loads by themselves, so that several degrees' are in flight)
#pragma unroll 4
  for (int L = aM; L <= S.Lmax; ++L) {
    const double d = __ldg(S.dL + L) * __ldg(p + L * (L + 1) / 2), f = (L & 2) ? -d : d;
    const double2 s = __ldg(sg + L * L + L + M);
    acc[0].x = fma(f, s.x, acc[0].x);
    acc[0].y = fma(f, s.y, acc[0].y);
    F[(size_t)L * nh * nM] = acc[0];
    const double2 x = acc[0];  // the two parities in turn
    acc[0] = acc[1];
    acc[1] = x;
  }
}

// Block: (l, m >= 0); thread: (l', m' >= 0) from (l, m) on, and the entries with
// both exchanged (the same integrals, F_M for F_-M).  The integrand is even: half
// the nodes.  Stored transposed, row l'm', columns lm (real part) and Kp + lm
// (imaginary part).  Bound by the reads of F through L2.
#define SMT_TH 64
__global__ void __launch_bounds__(SMT_TH) k_sm_T(const __grid_constant__ sm_dev S) {
  const int b = blockIdx.z;
  auto lm = [](int i, int &l, int &m) {
    l = (int)((sqrt(8.0 * i + 1.0) - 1.0) * 0.5);
    while ((l + 1) * (l + 2) / 2 <= i) ++l;
    while (l * (l + 1) / 2 > i) --l;
    m = i - l * (l + 1) / 2;
  };
  const int i1 = blockIdx.x, i2 = blockIdx.y * SMT_TH + threadIdx.x;
  const int nlm = (S.lmax + 1) * (S.lmax + 2) / 2;
  if (i2 < i1 || i2 >= nlm) return;
  int l, m, l2, m2;
  lm(i1, l, m);
  lm(i2, l2, m2);
  const int nM = 2 * S.Mx + 1, nh = S.nt / 2, sum = l + l2;
  const int j = sum <= S.Lmax ? sum : S.Lmax - ((S.Lmax ^ sum) & 1);
  const int M1 = m - m2, M2 = m + m2;
  const bool on2 = m && m2 && M2 <= S.Mx, on1 = abs(M1) <= S.Mx;
  const double2 *F = reinterpret_cast<const double2 *>(S.F) + ((size_t)b * (S.Lmax + 1) + j) * nh * nM + S.Mx;
  const double2 *Fa = F + (on1 ? M1 : 0), *Fb = F - (on1 ? M1 : 0), *Fc = F + (on2 ? M2 : 0), *Fd = F - (on2 ? M2 : 0);
  const double *p1 = S.plm + i1, *p2 = S.plm + i2;
  // tp[0]: T_{m,m'}, tp[1]: T_{-m,-m'}, tp[2]: T_{m,-m'}, tp[3]: T_{-m,m'}
  cplx tp[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) tp[c] = cmk(0.0, 0.0);
#pragma unroll 4
  for (int t = 0; t < nh; ++t) {
    const double pr = 4.0 * CUDART_PI * S.w[t] * p1[(size_t)t * S.nlm] * p2[(size_t)t * S.nlm];
    const size_t o = (size_t)t * nM;
    const double2 fa = Fa[o], fb = Fb[o], fc = Fc[o], fd = Fd[o];
    tp[0].re = fma(pr, fa.x, tp[0].re);
    tp[0].im = fma(pr, fa.y, tp[0].im);
    tp[1].re = fma(pr, fb.x, tp[1].re);
    tp[1].im = fma(pr, fb.y, tp[1].im);
    tp[2].re = fma(pr, fc.x, tp[2].re);
    tp[2].im = fma(pr, fc.y, tp[2].im);
    tp[3].re = fma(pr, fd.x, tp[3].re);
    tp[3].im = fma(pr, fd.y, tp[3].im);
  }
  if (!on1) tp[0] = tp[1] = cmk(0.0, 0.0);
  if (!on2) tp[2] = tp[3] = cmk(0.0, 0.0);
  // i^{l - l'} beside F's i^{-L}: even exponents together
  const double sc = 4.0 * CUDART_PI * S.el[l] * S.el[l2];
  sm_put_T(S, b, l, m, l2, m2, tp, ((l - l2) & 2) ? -sc : sc);
  if (i2 == i1) return;
  const cplx x = tp[0];
  tp[0] = tp[1];
  tp[1] = x;
  sm_put_T(S, b, l2, m2, l, m, tp, ((l2 - l) & 2) ? -sc : sc);
}

// ------------------------------------------------------------------ functions at nodes and over elements
// g_l(z), l = 0 .. n + 1, into g[l * stride] by downward recurrence
__device__ __forceinline__ void sm_gl(int n, double z2, double *g, int stride) {
  const int top = n + 1;
  double a = 0.0, b = 0.0;
#pragma unroll 1
  for (int w = 0; w < 2; ++w) {
    const int l = top + 1 - w;
    double t = 1.0, s = 1.0;
    for (int m = 1; m < 100; ++m) {
      t *= -0.5 * z2 / (m * (2.0 * l + 2.0 * m + 1.0));
      s += t;
      if (fabs(t) < 1e-18 * fabs(s)) break;
    }
    if (w == 0) a = s;
    else b = s;
  }
  g[top * stride] = b;  // g_top, a = g_{top + 1}
  for (int l = top; l > 0; --l) {
    const double c = b - z2 / ((2.0 * l + 1.0) * (2.0 * l + 3.0)) * a;
    a = b;
    b = c;
    g[(l - 1) * stride] = c;
  }
}

// U[p][lm] = phi_lm(x_p): a warp per node, a lane per order m
#define SMU_TH 128
__global__ void __launch_bounds__(SMU_TH) k_sm_targets(const __grid_constant__ sm_dev S, bem_dom_dev D) {
  __shared__ double g[SMU_TH / 32][BEM_SM_MAXL + 2];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * (SMU_TH / 32) + wid;
  if (p >= 4 * D.ne) return;
  const int te = abs(D.sid[p >> 2]) - 1;
  double *U = S.U + (size_t)p * S.Kp;
  const bool pad = (p & 3) == 3 && D.has_tri && D.npe[te] == 3;
  if (pad) {
    for (int c = lane; c < S.Kp; c += 32) U[c] = 0.0;
    return;
  }
  for (int c = S.K + lane; c < S.Kp; c += 32) U[c] = 0.0;
  const double *r = D.ren + (size_t)te * 12 + (p & 3) * 3;
  const double x = (r[0] - S.cx) * S.iR0, y = (r[1] - S.cy) * S.iR0, z = (r[2] - S.cz) * S.iR0;
  const double s2 = x * x + y * y + z * z;
  if (lane == 0) sm_gl(S.lmax, S.kR0 * S.kR0 * s2, g[wid], 1);
  __syncwarp();
  for (int m = lane; m <= S.lmax; m += 32) {
    double C = 1.0, Sn = 0.0;  // Re, Im (x + iy)^m
    for (int a = 0; a < m; ++a) {
      const double c2 = C * x - Sn * y;
      Sn = C * y + Sn * x;
      C = c2;
    }
    if (m) { C *= 1.4142135623730950488; Sn *= 1.4142135623730950488; }
    double t1 = S.rec[m * (m + 1) + 2 * m], t0 = 0.0;
    for (int l = m; l <= S.lmax; ++l) {
      if (l > m) {
        const double *rr = S.rec + l * (l + 1) + 2 * m;
        const double t2 = rr[0] * (z * t1 - rr[1] * s2 * t0);
        t0 = t1;
        t1 = t2;
      }
      const double v = g[wid][l] * t1;
      U[sm_idx(l, m, 0)] = v * C;
      if (m) U[sm_idx(l, m, 1)] = v * Sn;
    }
  }
}

// The values of order m at a point (r, W): for each degree l the rows |W| phi and
// W . grad phi of the cosine (and of the sine) function, SMV_PT apart, at val.
#define SMV_PT (BEM_GLN * BEM_GLN)
// shared memory of a kernel that keeps these values, rows more per point beside them
static int sm_point_smem(int rows, int lmax) {
  return (rows + std::max(2 * (lmax + 1), 4 * lmax)) * SMV_PT * (int)sizeof(double);
}
__device__ __forceinline__ void sm_point_values(const sm_dev &S, int m, int nf, const double r[3], const double W[3],
                                                double *val) {
        const double aW = sqrt(W[0] * W[0] + W[1] * W[1] + W[2] * W[2]);
        const double x = (r[0] - S.cx) * S.iR0, y = (r[1] - S.cy) * S.iR0, z = (r[2] - S.cz) * S.iR0;
        const double s2 = x * x + y * y + z * z;
        const double wx = W[0] * S.iR0, wy = W[1] * S.iR0, wz = W[2] * S.iR0;
        const double wr = wx * x + wy * y + wz * z;
        // Re, Im (x + iy)^m and their derivatives along W
        double C = 1.0, Sn = 0.0, C0 = 0.0, S0 = 0.0;
        for (int a = 0; a < m; ++a) {
          C0 = C;
          S0 = Sn;
          const double c2 = C * x - Sn * y;
          Sn = C * y + Sn * x;
          C = c2;
        }
        double dC = m * (wx * C0 - wy * S0), dS = m * (wx * S0 + wy * C0);
        if (m) {
          const double q2 = 1.4142135623730950488;
          C *= q2; Sn *= q2; dC *= q2; dS *= q2;
        }
        // g_l downward from l = lmax + 1, kept in the value slots until used
        const double z2 = S.kR0 * S.kR0 * s2, kk2 = S.kR0 * S.kR0;
        // upward walk needs g_l and g_{l+1}: g is computed into val[l - m][0]
        // (read before it is overwritten) with g_{lmax + 1} kept in a register
        double gtop;
        {
          double a = 0.0, b = 0.0;
  #pragma unroll 1
          for (int w = 0; w < 2; ++w) {
            const int l = S.lmax + 2 - w;
            double t = 1.0, sum = 1.0;
            for (int q = 1; q < 100; ++q) {
              t *= -0.5 * z2 / (q * (2.0 * l + 2.0 * q + 1.0));
              sum += t;
              if (fabs(t) < 1e-18 * fabs(sum)) break;
            }
            if (w == 0) a = sum;
            else b = sum;
          }
          gtop = b;
          for (int l = S.lmax + 1; l > m; --l) {
            const double c = b - z2 / ((2.0 * l + 1.0) * (2.0 * l + 3.0)) * a;
            a = b;
            b = c;
            val[(size_t)(l - 1 - m) * 2 * nf * SMV_PT] = c;
          }
        }
        double t1 = S.rec[m * (m + 1) + 2 * m], t0 = 0.0;  // Theta
        double p1 = 0.0, p0 = 0.0, q1 = 0.0, q0 = 0.0;     // dTheta/dz, dTheta/ds
        for (int l = m; l <= S.lmax; ++l) {
          if (l > m) {
            const double *rr = S.rec + l * (l + 1) + 2 * m;
            const double ra = rr[0], rb = rr[1];
            const double t2 = ra * (z * t1 - rb * s2 * t0);
            const double p2 = ra * (t1 + z * p1 - rb * s2 * p0);
            const double q2 = ra * (z * q1 - rb * (t0 + s2 * q0));
            t0 = t1; t1 = t2;
            p0 = p1; p1 = p2;
            q0 = q1; q1 = q2;
          }
          double *v = val + (size_t)(l - m) * 2 * nf * SMV_PT;
          const double g = v[0], gn = l < S.lmax ? v[2 * nf * SMV_PT] : gtop;
          // W . grad (g Theta C) = [g (wz P + 2 wr Q) - wr kk^2 g_{l+1} / (2l + 3) Theta] C + g Theta W . grad C
          const double gt = g * t1;
          const double f = g * (wz * p1 + 2.0 * wr * q1) - wr * kk2 * gn / (2.0 * l + 3.0) * t1;
          v[0] = aW * gt * C;
          v[SMV_PT] = f * C + gt * dC;
          if (nf == 2) {
            v[2 * SMV_PT] = aW * gt * Sn;
            v[3 * SMV_PT] = f * Sn + gt * dS;
          }
        }
}

// V[lm][4 s + a] = int N_a |W| phi_lm, V[lm][4 ne + 4 s + a] = int N_a W . grad phi_lm
// over element s.  The product with A makes these G_s and W . grad G_s integrated
// with this rule, so the rule is the one a regular pair takes whose nearest image
// is at the least distance any image left in has from an element (cut - 2 R0);
// the reference's 12 x 12 (3 parts of it on a triangle) without the shorter rules.  Block: (element, order m); a thread per point walks l and leaves
// the four values of each l in shared memory, then a thread per value sums
// over the points.
#define SMV_TH 160
__global__ void __launch_bounds__(SMV_TH) k_sm_sources(const __grid_constant__ sm_dev S, bem_dom_dev D, int far_rule) {
  extern __shared__ double sm_raw[];
  const int s = blockIdx.x, m = blockIdx.y, tid = threadIdx.x;
  const int se = abs(D.sid[s]) - 1;
  const bool tri = D.has_tri && D.npe[se] == 3;
  const int nl = S.lmax + 1 - m, nf = m ? 2 : 1;  // functions per degree
  double *Nw = sm_raw;                  // [4][SMV_PT] weight times N_a
  double *val = Nw + 4 * SMV_PT;        // [nl][2 nf][SMV_PT]
  const int nout = nl * 2 * nf;
  const size_t N8 = 8 * (size_t)D.ne;
  double acc[4] = {0, 0, 0, 0};
  bem_el el;
  bem_load_el(D.cr, D.cw, se, el);
  int tier = -1;
  if (far_rule) {
    const double R2 = el_circum2(el, tri);
    tier = tier_image(S.cut * S.cut / R2, S.k * S.k * R2, tri, tri || quad_tier_shape(el));
  }
  const int n = tier < 0 ? BEM_GLN : BEM_TIER_N0 - tier, npt = n * n;
  for (int part = 0; part < (tri && tier < 0 ? 3 : 1); ++part) {
    if (part) __syncthreads();
    if (tid < npt) {
      double zt, et, wt;
      rule_pt(n, tri, part * npt + tid, zt, et, wt);
      double r[3], W[3], Nn[4];
      bem_rw(el, zt, et, r, W);
      bem_Nn(tri, zt, et, Nn);
#pragma unroll
      for (int a = 0; a < 4; ++a) Nw[a * SMV_PT + tid] = Nn[a] * wt;
      sm_point_values(S, m, nf, r, W, val + tid);
    }
    __syncthreads();
    if (tid < nout) {
      const double *v = val + (size_t)tid * SMV_PT;
      const int q0 = tid % npt;  // another first point per thread: the rows are a multiple of 32 banks apart
      for (int q = 0; q < npt; ++q) {
        const int qq = q + q0 < npt ? q + q0 : q + q0 - npt;
        const double x = v[qq];
#pragma unroll
        for (int a = 0; a < 4; ++a) acc[a] = fma(x, Nw[a * SMV_PT + qq], acc[a]);
      }
    }
  }
  if (tid < nout) {
    const int l = m + tid / (2 * nf), r = tid % (2 * nf);  // r: value, derivative (, sine value, derivative)
    double *o = S.V + (size_t)sm_idx(l, m, r >> 1) * N8 + ((r & 1) ? 4 * (size_t)D.ne : 0) + 4 * (size_t)s;
#pragma unroll
    for (int a = 0; a < 4; ++a) o[a] = acc[a];
  }
  if (m == 0 && tid < 8)  // padding rows of V
    for (int r = S.K; r < S.Kp; ++r)
      S.V[(size_t)r * N8 + (tid < 4 ? 0 : 4 * (size_t)D.ne) + 4 * (size_t)s + (tid & 3)] = 0.0;
}

// ------------------------------------------------------------------ real matrix product on the FP64 tensor cores
// C = A B, A M x K (row-major, lda), B K x N (row-major, ldb), K a multiple of
// 16, lda and ldb even.  128 x 64 tiles, 8 warps of 32 x 32, mma m16n8k8,
// operands through a 3-stage ring of 16-deep slices filled by 16-byte
// asynchronous copies; row strides of 20 and 68 doubles keep the fragment
// loads free of bank conflicts.  ILV: rows 2p and 2p + 1 are the real and
// imaginary parts of row p of a complex result whose columns below N / 2 go to
// G and the others to H (leading dimension N / 2).
#define GM_BM 128
#define GM_BN 64
#define GM_BK 16
#define GM_ST 3
#define GM_LDA 20
#define GM_LDB 68
#define GM_TH 256
#define GM_STAGE (GM_BM * GM_LDA + GM_BK * GM_LDB)
#define GM_SMEM (GM_ST * GM_STAGE * 8)
__device__ __forceinline__ void gm_cp16(double *dst, const double *src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void gm_mma(const double (&a)[4], const double (&b)[2], double (&d)[4]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
template <bool ILV>
__global__ void __launch_bounds__(GM_TH, 2) k_sm_gemm(const double *A0, size_t strideA, int lda, const double *B0,
                                                      size_t strideB, int ldb, int M, int N, int K, double *C0,
                                                      size_t strideC, int ldc, const __grid_constant__ sm_out O) {
  extern __shared__ __align__(16) double gm_smem[];
  const double *A = A0 + blockIdx.z * strideA, *B = B0 + blockIdx.z * strideB;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, g = lane >> 2, q = lane & 3;
  const int rb = blockIdx.y * GM_BM, cb = blockIdx.x * GM_BN;
  const int wm = (wid & 3) * 32, wn = (wid >> 2) * 32;
  auto fill = [&](int st, int k0) {
    double *As = gm_smem + st * GM_STAGE, *Bs = As + GM_BM * GM_LDA;
#pragma unroll
    for (int i = 0; i < GM_BM * GM_BK / 2 / GM_TH; ++i) {
      const int e = t + i * GM_TH, r = e >> 3, c = (e & 7) * 2;
      const bool live = rb + r < M;
      gm_cp16(As + r * GM_LDA + c, A + (size_t)(live ? rb + r : 0) * lda + k0 + c, live);
    }
#pragma unroll
    for (int i = 0; i < GM_BK * GM_BN / 2 / GM_TH; ++i) {
      const int e = t + i * GM_TH, r = e >> 5, c = (e & 31) * 2;
      const bool live = cb + c < N;
      gm_cp16(Bs + r * GM_LDB + c, B + (size_t)(k0 + r) * ldb + (live ? cb + c : 0), live);
    }
  };
  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0;
  const int nk = K / GM_BK;
#pragma unroll
  for (int s = 0; s < GM_ST - 1; ++s) {
    if (s < nk) fill(s, s * GM_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GM_ST - 2) : "memory");
    __syncthreads();  // slice kt is in, and every warp is done with slice kt - 1
    if (kt + GM_ST - 1 < nk) fill((kt + GM_ST - 1) % GM_ST, (kt + GM_ST - 1) * GM_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double *As = gm_smem + (kt % GM_ST) * GM_STAGE, *Bs = As + GM_BM * GM_LDA;
#pragma unroll
    for (int k8 = 0; k8 < GM_BK; k8 += 8) {
      double a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) a[i][c] = As[(wm + i * 16 + g + (c & 1) * 8) * GM_LDA + k8 + q + (c >> 1) * 4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) b[j][c] = Bs[(k8 + q + c * 4) * GM_LDB + wn + j * 8 + g];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) gm_mma(a[i], b[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = rb + wm + i * 16 + g + 8 * h, col = cb + wn + j * 8 + 2 * q;
        const double d0 = acc[i][j][2 * h], d1 = acc[i][j][2 * h + 1];
        if (!ILV) {
          if (row < M && col < N)
            *reinterpret_cast<double2 *>(C0 + blockIdx.z * strideC + (size_t)row * ldc + col) = make_double2(d0, d1);
        } else {
          // the lane four away holds the other part of the same row of G, H:
          // the even row's lane takes column col, the odd row's col + 1
          const bool odd = g & 1;
          const double other = __shfl_xor_sync(0xffffffffu, odd ? d0 : d1, 4);
          const int cc = col + (odd ? 1 : 0), N2 = N / 2;
          const double2 z = odd ? make_double2(other, d1) : make_double2(d0, other);
          if (row < M && cc < N) {
            double *dst = (cc < N2 ? O.G[blockIdx.z] : O.H[blockIdx.z]) + 2 * ((size_t)(row >> 1) * N2 + (cc < N2 ? cc : cc - N2));
            *reinterpret_cast<double2 *>(dst) = z;
          }
        }
      }
}

// ------------------------------------------------------------------ images
// The images of every pair off the lattice plane, in closed form, added to G
// and H: LP lanes per pair, each a share of the rule's points.  The home
// image of a regular pair takes the pair's own rule (its flag); the others
// share the points of the rule for the nearest of them, so that an element's
// geometry is formed once for all.  A warp takes the longest rule its pairs
// ask for.  FP64 pipe: about 66 operations per image and point.
#define SMI_TH 128
template <int LP>
__global__ void __launch_bounds__(SMI_TH, 4) k_sm_images(const __grid_constant__ sm_dev S, bem_dom_dev D, int far_rule,
                                                         const uint8_t *__restrict__ flag,
                                                         const __grid_constant__ sm_out O) {
  __shared__ double im[3 * BEM_SM_MAXIMG];
  const int b = blockIdx.y;
  for (int e = threadIdx.x; e < 3 * S.nimg; e += SMI_TH) im[e] = S.img[3 * b * S.nimg + e];
  __syncthreads();
  const long long npairs = 4LL * D.ne * D.ne;
  const long long pair = ((long long)blockIdx.x * SMI_TH + threadIdx.x) / LP;
  const int sub = threadIdx.x % LP;
  const bool in = pair < npairs;
  const int p = in ? (int)(pair / D.ne) : 0, s = in ? (int)(pair % D.ne) : 0;
  const int fl = in ? flag[pair] : 0;
  const int te = abs(D.sid[p >> 2]) - 1, se = abs(D.sid[s]) - 1;
  const bool tri = D.has_tri && __ldg(D.npe + se) == 3;
  const bool live = in && fl != 0 && !((p & 3) == 3 && D.has_tri && __ldg(D.npe + te) == 3);
  bem_el el;
  bem_load_el(D.cr, D.cw, se, el);
#pragma unroll
  for (int d = 0; d < 3; ++d) el.cr[d][0] -= __ldg(D.ren + (size_t)te * 12 + (p & 3) * 3 + d);  // r is R now
  int n1 = 0, n2 = 0;
  if (live) {
    if (fl >= 3) n1 = fl == BEM_FL_REF ? BEM_GLN : BEM_TIER_N0 - (fl - 3);
    n2 = BEM_GLN;
    if (far_rule && S.nimg > 1) {
      double d2 = 1e300;
      for (int m = 1; m < S.nimg; ++m) {
        const double x = el.cr[0][0] + im[3 * m], y = el.cr[1][0] + im[3 * m + 1];
        d2 = fmin(d2, fma(x, x, y * y));
      }
      d2 = fma(el.cr[2][0], el.cr[2][0], d2);
      const double R2 = el_circum2(el, tri);
      const int t = tier_image(d2 / R2, S.k * S.k * R2, tri, tri || quad_tier_shape(el));
      if (t >= 0) n2 = BEM_TIER_N0 - t;
    }
    if (S.nimg == 1) n2 = 0;
  }
  const int w1 = __reduce_max_sync(0xffffffffu, n1);
  n1 = n1 ? w1 : 0;
  n2 = __reduce_max_sync(0xffffffffu, n2);
  double v[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) v[c] = 0.0;
  const double k = S.k, kpi = S.k * 0.31830988618379067154;
#pragma unroll 1
  for (int grp = 0; grp < 2; ++grp) {
    if (grp == 0 ? n1 == 0 : (!live || n2 == 0)) continue;
    const int n = grp == 0 ? n1 : n2;
    const int m0 = grp, m1 = grp == 0 ? 1 : S.nimg, np = rule_npts(n, tri);
#pragma unroll 1
    for (int pt = sub; pt < np; pt += LP) {
      double z, e, wt;
      rule_pt(n, tri, pt, z, e, wt);
      double R[3], W[3];
      bem_rw(el, z, e, R, W);
      const double rz2 = R[2] * R[2], rzw = R[2] * W[2];
      double gr = 0.0, gi = 0.0, hr = 0.0, hi = 0.0;
#pragma unroll 2
      for (int m = m0; m < m1; ++m) {
        const double px = R[0] + im[3 * m], py = R[1] + im[3 * m + 1];
        double a, c, fr, fi;
        sm_image(kpi, k, px, py, rz2, im[3 * m + 2], a, c, fr, fi);
        const double dw = fma(px, W[0], fma(py, W[1], rzw));
        gr += a;
        gi += c;
        hr = fma(fr, dw, hr);
        hi = fma(fi, dw, hi);
      }
      const double aw = sqrt(W[0] * W[0] + W[1] * W[1] + W[2] * W[2]) * wt;
      gr *= aw; gi *= aw; hr *= wt; hi *= wt;
      double N[4];
      bem_Nn(tri, z, e, N);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        v[2 * a] = fma(gr, N[a], v[2 * a]);
        v[2 * a + 1] = fma(gi, N[a], v[2 * a + 1]);
        v[8 + 2 * a] = fma(hr, N[a], v[8 + 2 * a]);
        v[8 + 2 * a + 1] = fma(hi, N[a], v[8 + 2 * a + 1]);
      }
    }
  }
#pragma unroll
  for (int o = LP / 2; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] += __shfl_down_sync(0xffffffffu, v[c], o, LP);
  if (live && sub == 0) {
    const size_t at = (size_t)p * (4 * (size_t)D.ne) + 4 * (size_t)s;
    double2 *G = reinterpret_cast<double2 *>(O.G[b]) + at, *H = reinterpret_cast<double2 *>(O.H[b]) + at;
    const int na = tri ? 3 : 4;
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if (a < na) {
        double2 x = G[a], y = H[a];
        x.x = fma(BEM_I_FP, v[2 * a], x.x);
        x.y = fma(BEM_I_FP, v[2 * a + 1], x.y);
        y.x = fma(BEM_I_FP, v[8 + 2 * a], y.x);
        y.y = fma(BEM_I_FP, v[8 + 2 * a + 1], y.y);
        G[a] = x;
        H[a] = y;
      }
  }
}

// ------------------------------------------------------------------ launches
// instances b0, b0 + 1, ... of the tables; held: sigma and T of instance b0 where
// the last launch_rest left them (otherwise at the front, where it will put them)
static sm_dev dev_view(const bem_smooth *S, int ne, int b0, bool held = false) {
  sm_dev d;
  d.lmax = S->lmax; d.Lmax = S->Lmax; d.K = S->K; d.Kp = S->Kp; d.nt = S->nt; d.nphi = S->nphi; d.nimg = S->nimg;
  d.eta = S->eta;
  d.r1 = S->r1; d.r2 = S->r2; d.nreal = (2 * S->r1 + 1) * (2 * S->r2 + 1);
  d.s1 = S->s1; d.s2 = S->s2; d.nspec = (2 * S->s1 + 1) * (2 * S->s2 + 1);
  for (int i = 0; i < S->nimg; ++i) { d.iml[2 * i] = S->l1[i]; d.iml[2 * i + 1] = S->l2[i]; }
  d.nlm = (S->Lmax + 1) * (S->Lmax + 2) / 2;
  d.cx = S->ctr[0]; d.cy = S->ctr[1]; d.cz = S->ctr[2];
  d.R0 = S->R0; d.iR0 = 1.0 / S->R0; d.kR0 = S->k * S->R0; d.rho = S->rho; d.k = S->k; d.cut = S->cut;
  const bem_smooth_tab t = bem_smooth_layout(S);
  d.x = S->tab + t.x; d.w = S->tab + t.w; d.ca = S->tab + t.ca; d.cb = S->tab + t.cb;
  d.dL = S->tab + t.dL; d.el = S->tab + t.el; d.rec = S->tab + t.rec;
  d.img = S->tab + t.img + 3 * (size_t)b0 * S->nimg;
  const sm_keep k = keep_layout(S);
  const size_t at = held ? b0 - S->have0 : 0;
  for (int i = 0; i < 8; ++i) d.lcut[i] = S->lcut[i];
  d.plm = S->keep + k.plm;
  d.samp = S->keep + k.samp;
  d.sig = S->keep + k.sig + at * 2 * (S->Lmax + 1) * (S->Lmax + 1);
  d.Mx = std::min(2 * S->lmax, S->Lmax);
  d.F = S->keep + k.F;
  d.T = S->keep + k.T + at * 2 * S->Kp * S->Kp;
  d.Z = S->keep + k.Z;
  d.Zt = S->keep + k.Zt;
  const sm_ws w = ws_layout(S, ne);
  d.U = S->ws + w.U;
  d.V = S->ws + w.V;
  d.A = S->ws + w.A;
  return d;
}

// sigma and T of n <= BEM_SM_BAT instances from instance b0 on
static int launch_rest(bem_smooth *S, const bem_qp *qps, int b0, int n, unsigned *status, cudaStream_t st) {
  const sm_dev d = dev_view(S, 0, b0);
  sm_qps Q;
  for (int i = 0; i < BEM_SM_BAT; ++i) Q.q[i] = qps[i < n ? i : 0];
  const int nlm = (S->lmax + 1) * (S->lmax + 2) / 2;
  const int nsamp = (S->nt * S->nphi * 32 + SMP_TH - 1) / SMP_TH, nleg = ((S->Lmax + 1) * S->nt + SMP_TH - 1) / SMP_TH;
  S->have0 = S->have1 = 0;
  k_sm_sample<<<dim3(nsamp + nleg, n), SMP_TH, 0, st>>>(d, Q, nsamp, status);
  k_sm_coef<<<dim3(2 * S->Lmax + 1, n), SMC_TH, 0, st>>>(d);
  k_sm_F<<<dim3(((2 * d.Mx + 1) * (S->nt / 2) + SMF_FTH - 1) / SMF_FTH, n), SMF_FTH, 0, st>>>(d);
  if (cudaMemsetAsync(d.T, 0, (size_t)n * 2 * S->Kp * S->Kp * sizeof(double), st) != cudaSuccess) return -1;
  k_sm_T<<<dim3(nlm, (nlm + SMT_TH - 1) / SMT_TH, n), SMT_TH, 0, st>>>(d);
  bem_count_launches(4);
  if (cudaPeekAtLastError() != cudaSuccess) return -1;
  S->have0 = b0;
  S->have1 = b0 + n;
  return 0;
}

template <int LP>
static void launch_images(const sm_dev &d, const bem_dom_dev *D, int nb, const uint8_t *flag, const sm_out &O, cudaStream_t st) {
  const long long th = 4LL * D->ne * D->ne * LP;
  k_sm_images<LP><<<dim3((unsigned)((th + SMI_TH - 1) / SMI_TH), nb), SMI_TH, 0, st>>>(d, *D, D->far_rule, flag, O);
}

extern "C" int bem_launch_smooth(bem_smooth *S, const bem_dom_dev *D, const bem_qp *qps, int nb, double *const *G,
                                 double *const *H, const bem_scratch *scr, cudaStream_t st) {
  const int ne = D->ne, N = 4 * ne;
  const int smem_v = sm_point_smem(4, S->lmax);
  const long long npairs = (long long)N * ne;
  for (int b0 = 0; b0 < nb; b0 += BEM_SM_BAT) {
    const int n = nb - b0 < BEM_SM_BAT ? nb - b0 : BEM_SM_BAT;
    const int first = nb == 1 ? S->first : b0;
    if (launch_rest(S, qps + b0, first, n, scr->status, st)) return -1;
    const sm_dev d = dev_view(S, ne, first);
    sm_out O;
    for (int i = 0; i < BEM_SM_BAT; ++i) {
      O.G[i] = i < n ? G[b0 + i] : nullptr;
      O.H[i] = i < n ? H[b0 + i] : nullptr;
    }
    if (b0 == 0) {
      k_sm_targets<<<(N + SMU_TH / 32 - 1) / (SMU_TH / 32), SMU_TH, 0, st>>>(d, *D);
      k_sm_sources<<<dim3(ne, S->lmax + 1), SMV_TH, smem_v, st>>>(d, *D, D->far_rule);
      bem_count_launches(2);
    }
    const size_t sT = 2 * (size_t)S->Kp * S->Kp, sA = (size_t)N * 2 * S->Kp;
    k_sm_gemm<false><<<dim3((2 * S->Kp + GM_BN - 1) / GM_BN, (N + GM_BM - 1) / GM_BM, n), GM_TH, GM_SMEM, st>>>(
        d.U, 0, S->Kp, d.T, sT, 2 * S->Kp, N, 2 * S->Kp, S->Kp, d.A, sA, 2 * S->Kp, O);
    k_sm_gemm<true><<<dim3((8 * ne + GM_BN - 1) / GM_BN, (2 * N + GM_BM - 1) / GM_BM, n), GM_TH, GM_SMEM, st>>>(
        d.A, sA, S->Kp, d.V, 0, 8 * ne, 2 * N, 8 * ne, S->Kp, nullptr, 0, 0, O);
    // Lanes per pair: 32 where a thread a pair leaves most of the GPU's 75,000 resident
    // threads idle, then 4, 1 where pairs alone are many waves and a lane's share of a
    // short rule gets small.  Measured, us with 32 / 4 / 1 lanes (square lattice, period
    // 0.8): 24 quads (2304 pairs) 37 / 117 / 440, 80 triangles (25,600) 192 / 451 / 1123, 96
    // quads (36,864) 213 / 192 / 371, 216 (186,624) 958 / 672 / 799, 600 (1.44e6) 7117 / 3711 /
    // 3824, 726 (2.1e6) 8152 / 3849 / 3884, 1014 (4.1e6) 16178 / 7212 / 7038, 1536 (9.4e6) 36612
    // / 15878 / 15099.  The lines lie where quads and triangles together lose least below
    // (32 to 4) and where 4 and 1 are within 3 % of each other on quads; 1280 triangles
    // (6.6e6) would take 9441 with 4 for 10902.
    const long long work = npairs * n;
    if (work >= 1500000) launch_images<1>(d, D, n, scr->flag, O, st);
    else if (work >= 60000) launch_images<4>(d, D, n, scr->flag, O, st);
    else launch_images<32>(d, D, n, scr->flag, O, st);
    bem_count_launches(3);
  }
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

#include "bem_bdsum.cuh"
#include "bem_smfield.cuh"

// The attributes belong to the device's functions, not to a context: every context sets
// the same, the most that any degree takes, so that threads with bodies of different
// degrees leave each other's launches valid.
extern "C" int bem_smooth_set_constants(const void *quad, const void *wc) {
  const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if (cudaMemcpyToSymbol(c_q, quad, sizeof(bem_quad)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_w, wc, sizeof(bem_wconst)) != cudaSuccess ||
      cudaFuncSetAttribute(k_sm_sources, at, sm_point_smem(4, BEM_SM_MAXL)) != cudaSuccess ||
      cudaFuncSetAttribute(k_sm_density, at, sm_point_smem(16, BEM_SM_MAXL)) != cudaSuccess ||
      cudaFuncSetAttribute(k_sm_gemm<true>, at, GM_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(k_sm_gemm<false>, at, GM_SMEM) != cudaSuccess)
    return -1;
  return 0;
}
