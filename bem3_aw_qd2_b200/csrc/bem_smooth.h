// The quasi-periodic Green's function of the host domain split into a few
// lattice images and a smooth rest (bem_smooth.cu).
#pragma once
#include <cuda_runtime.h>
#include "bem_kernels.h"

#define BEM_SM_MAXL 40     // largest degree of the expansion about the body's centre
#define BEM_SM_MAXIMG 40   // most lattice images taken out
#define BEM_SM_BAT 8       // instances per launch

// The split of one body and lattice: which images are taken out, and the
// degrees that represent the rest to FP64 round-off.  Host data; tab is what
// the device needs of it.
struct bem_smooth {
  int on = 0;
  int lmax = 0, Lmax = 0, K = 0, Kp = 0, nt = 0, nphi = 0, nimg = 0;
  double ctr[3] = {0, 0, 0}, R0 = 0.0, rho = 0.0, k = 0.0;
  double cut = 0.0;             // least distance of an image left in from an element, seen from a node
  double eta = 0.0;             // Ewald parameter and windows of the samples
  int r1 = 0, r2 = 0, s1 = 0, s2 = 0;
  int l1[BEM_SM_MAXIMG], l2[BEM_SM_MAXIMG];  // the images' lattice indices, (0, 0) first
  int np = 0;                   // the nearest lattice points, by distance (as many as a split
  double pr[BEM_SM_MAXIMG + 1]; // can look at: its images and the first shell left in)
  int p1[BEM_SM_MAXIMG + 1], p2[BEM_SM_MAXIMG + 1];
  int inst = 1, first = 0;      // instances tab holds; the one a launch for a single instance takes
  const double *tab = nullptr;  // device copy of the tables bem_smooth_tables writes
  int lcut[8] = {};             // degrees of the expansion about a point, by distance (boundary sums; not a field's plan)
  double *keep = nullptr;       // device memory of bem_smooth_keep_doubles doubles, kept with the problem
  int have0 = 0, have1 = 0;     // instances whose expansion keep holds
  double *ws = nullptr;         // an assembly's scratch, bem_smooth_ws_doubles doubles
};
// offsets (doubles) in tab
struct bem_smooth_tab {
  int x, w, ca, cb, dL, el, rec, img, total;
};

// Choose the images and degrees for the elements (cr, npe; ids sid[0 .. ne))
// of the periodic domain; S.on = 0 where the split does not pay (a body much
// taller or wider than the lattice period).
void bem_smooth_plan(bem_smooth *S, const bem_qp *q, const double *cr, const int *npe, const int *sid, int ne);
bem_smooth_tab bem_smooth_layout(const bem_smooth *S);
// the tables of S->inst instances (qps: their Bloch wave vectors) into h[layout.total]
void bem_smooth_tables(const bem_smooth *S, const bem_qp *qps, double *h);
// the split for sums at n points up to Rx from the body's centre; returns its operations,
// 1e300 where there is none of fewer than limit (then F->on = 0)
double bem_smooth_plan_field(bem_smooth *F, const bem_smooth *S, const bem_qp *q, double Rx, double n, double sources,
                             double limit);
size_t bem_smooth_keep_doubles(const bem_smooth *S);
size_t bem_smooth_ws_doubles(const bem_smooth *S, int ne);
// what a problem of ne elements allocates for its split (0 where it is off), doubles: the
// tables, what is kept, and the scratch of several instances or of one that is larger
// than the lent doubles (the global matrix, which holds nothing during an assembly)
struct bem_smooth_room { size_t tab, keep, ws; };
bem_smooth_room bem_smooth_need(const bem_smooth *S, int ne, size_t lent);

extern "C" {
// constant tables of this translation unit (quad: bem_quad, wc: bem_wconst) and its
// kernels' attributes, on the current device
int bem_smooth_set_constants(const void *quad, const void *wc);
// G, H of nb instances of the periodic domain: the smooth rest of every pair
// (written), then the images of every pair off the lattice plane (added; the
// home image of near-singular and self pairs is left to their own kernels)
int bem_launch_smooth(bem_smooth *S, const bem_dom_dev *D, const bem_qp *qps, int nb, double *const *G,
                      double *const *H, const bem_scratch *scr, cudaStream_t st);
// k_bdval's sums for targets of the periodic domain (bem_bdsum.cuh); q: the
// parameters of instance S->first
int bem_launch_bdsum(bem_smooth *S, const bem_dom_dev *D, const bem_qp *q, int type, int ntgt, const int *tgt_t,
                     const double *tgt_ze, const double *P, const double *dP, const double *pv, const double *dpv,
                     double *out, unsigned *status, cudaStream_t st);
// Field sums of k_field at points within the ball of a plan made by
// bem_smooth_plan_field (bem_smfield.cuh); pts, out as bem_launch_field's, again[i]: 1
// where a source lies on the lattice plane through point i (out not written)
int bem_launch_smfield(bem_smooth *F, const bem_dom_dev *D, const bem_qp *q, int grad, int type, int npts,
                       const double *pts, const double *P, const double *dP, const double *pv, const double *dpv,
                       double *out, int *again, unsigned *status, cudaStream_t st);
}
