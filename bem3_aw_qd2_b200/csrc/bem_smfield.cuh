// Field sums of the periodic domain (k_field, bem_post.cuh) with the images and the
// expansion of bem_smooth.cu, on a plan whose ball holds the points as well as the
// body; included at its end.  A lattice sum with second derivatives is some 1e4
// operations a pair; here a pair is 10 to 40 images of 160 (e^{ikR} / R, its
// gradient and its second derivatives along W), and the rest of all sources is one
// sum of K regular waves a point.  1500 points of 216 quads on the 9-point rule: 11.0
// ms with the tabled lattice sums of k_field, 1.54 ms like this, of which the sums
// take 1.02 (images, 40 % of the FP64 pipe's peak).  A
// point with a source on its lattice plane is left to k_field.
#pragma once

#define SMF_TH 128

__global__ void __launch_bounds__(SMF_TH) k_sm_field(const __grid_constant__ sm_dev S, bem_dom_dev D, int grad, int type,
                                                     const double *__restrict__ pts, const double *__restrict__ P,
                                                     const double *__restrict__ dP, const double *__restrict__ pv,
                                                     const double *__restrict__ dpv, double *__restrict__ out,
                                                     int *__restrict__ again) {
  __shared__ double im[3 * BEM_SM_MAXIMG], gl[BEM_SM_MAXL + 2];
  const int ip = blockIdx.x, tid = threadIdx.x;
  for (int e = tid; e < 3 * S.nimg; e += SMF_TH) im[e] = S.img[e];
  const double rt[3] = {pts[3 * ip], pts[3 * ip + 1], pts[3 * ip + 2]};
  const double tx = (rt[0] - S.cx) * S.iR0, ty = (rt[1] - S.cy) * S.iR0, tz = (rt[2] - S.cz) * S.iR0;
  const double ts2 = tx * tx + ty * ty + tz * tz, kk2 = S.kR0 * S.kR0;
  if (tid == SMF_TH - 1) sm_gl(S.lmax, kk2 * ts2, gl, 1);
  __syncthreads();
  const int nr = D.has_tri ? max(rule_points(type), tri_rule_points(type)) : rule_points(type);
  const int nit = D.ne * nr;
  const double kpi = S.k * 0.31830988618379067154;
  double a[18];
#pragma unroll
  for (int c = 0; c < 18; ++c) a[c] = 0.0;
  bool met = false;
  for (int it = tid; it < nit; it += SMF_TH) {
    const int s = it / nr, i = it % nr, se = abs(D.sid[s]) - 1;
    const bool stri = D.has_tri && D.npe[se] == 3;
    if (i >= (stri ? tri_rule_points(type) : rule_points(type))) continue;
    double z, e, w, vR[3], vW[3];
    bd_source_point(D, se, stri, type, i, z, e, w, vR, vW);
    for (int d = 0; d < 3; ++d) vR[d] = __dsub_rn(vR[d], rt[d]);
    met |= fabs(vR[2]) < BEM_FAR_PLANE_TOL;
    // images: value, gradient, second derivatives along W
    const double rz2 = vR[2] * vR[2], zw = vR[2] * vW[2];
    double g[2] = {0, 0}, f[6] = {0, 0, 0, 0, 0, 0}, fs[2] = {0, 0}, h[6] = {0, 0, 0, 0, 0, 0};
    for (int m = 0; m < S.nimg; ++m) {
      const double px = vR[0] + im[3 * m], py = vR[1] + im[3 * m + 1];
      const double r2 = fma(px, px, fma(py, py, rz2)), ir = rsqrt(r2), r = r2 * ir, ir2 = ir * ir, kr = S.k * r;
      double sn, cs;
      sincospi(fma(kpi, r, im[3 * m + 2]), &sn, &cs);
      const double gr = ir * cs, gi = ir * sn;
      const double fr = -ir2 * fma(kr, gi, gr), fi = ir2 * fma(kr, gr, -gi);
      g[0] += gr;
      g[1] += gi;
      f[0] = fma(fr, px, f[0]);
      f[1] = fma(fi, px, f[1]);
      f[2] = fma(fr, py, f[2]);
      f[3] = fma(fi, py, f[3]);
      fs[0] += fr;
      fs[1] += fi;
      if (grad) {
        // (3 - k^2 r^2 - 3 i k r) g / r^4, times P . W
        const double pw = fma(px, vW[0], fma(py, vW[1], zw)) * ir2 * ir2, u = 3.0 - kr * kr, v = 3.0 * kr;
        const double er = fma(u, gr, v * gi) * pw, ei = fma(u, gi, -v * gr) * pw;
        h[0] = fma(er, px, h[0]);
        h[1] = fma(ei, px, h[1]);
        h[2] = fma(er, py, h[2]);
        h[3] = fma(ei, py, h[3]);
        h[4] += er;
        h[5] += ei;
      }
    }
    f[4] = fs[0] * vR[2];
    f[5] = fs[1] * vR[2];
    h[4] *= vR[2];
    h[5] *= vR[2];
    cplx Pn, dPn, pvn[3], dpvn[3];
    interp_bv(type, i, z, e, s, P, dP, pv, dpv, Pn, dPn, pvn, dpvn, stri);
    const double wg = w * BEM_I_FP, aW = sqrt(dot3(vW, vW));
    const cplx G = cmk(wg * aW * g[0], wg * aW * g[1]);
    const cplx H = cmk(wg * (f[0] * vW[0] + f[2] * vW[1] + f[4] * vW[2]), wg * (f[1] * vW[0] + f[3] * vW[1] + f[5] * vW[2]));
    const cplx t0 = csub(cmul(G, dPn), cmul(H, Pn));
    a[0] += t0.re;
    a[1] += t0.im;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const cplx t2 = csub(cmul(G, dpvn[j]), cmul(H, pvn[j]));
      a[12 + 2 * j] += t2.re;
      a[13 + 2 * j] += t2.im;
      if (grad) {  // d / d rt = -d / d R
        const cplx dG = cmk(-wg * aW * f[2 * j], -wg * aW * f[2 * j + 1]);
        const cplx dH = cmk(-wg * (fs[0] * vW[j] + h[2 * j]), -wg * (fs[1] * vW[j] + h[2 * j + 1]));
        const cplx t1 = csub(cmul(dG, dPn), cmul(dH, Pn));
        a[2 + 2 * j] += t1.re;
        a[3 + 2 * j] += t1.im;
      }
    }
    fld_geom(vR, vW, D.sid[s] < 0 ? -w : w, a + 8);
  }
  met = __syncthreads_or(met);
  if (tid == 0) again[ip] = met;
  if (met) return;
  // the rest: sum_k phi_k(rt) Zt_k and the gradient of the potential's, a thread per order
  for (int m = tid; m <= S.lmax; m += SMF_TH) {
    double C = 1.0, Sn = 0.0, C0 = 0.0, S0 = 0.0;
    for (int b = 0; b < m; ++b) {
      C0 = C;
      S0 = Sn;
      const double c2 = C * tx - Sn * ty;
      Sn = C * ty + Sn * tx;
      C = c2;
    }
    if (m) { C *= 1.4142135623730950488; Sn *= 1.4142135623730950488; C0 *= 1.4142135623730950488; S0 *= 1.4142135623730950488; }
    double t1 = S.rec[m * (m + 1) + 2 * m], t0 = 0.0, p1 = 0.0, p0 = 0.0, q1 = 0.0, q0 = 0.0;
    for (int l = m; l <= S.lmax; ++l) {
      if (l > m) {
        const double *rr = S.rec + l * (l + 1) + 2 * m;
        const double ra = rr[0], rb = rr[1];
        const double t2 = ra * (tz * t1 - rb * ts2 * t0);
        const double p2 = ra * (t1 + tz * p1 - rb * ts2 * p0);
        const double q2 = ra * (tz * q1 - rb * (t0 + ts2 * q0));
        t0 = t1; t1 = t2;
        p0 = p1; p1 = p2;
        q0 = q1; q1 = q2;
      }
      const double v = gl[l] * t1, fz = gl[l] * p1, fr = 2.0 * gl[l] * q1 - kk2 * gl[l + 1] / (2.0 * l + 3.0) * t1;
      const double *zc = S.Zt + 8 * sm_idx(l, m, 0);
      double zs[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) zs[c] = m ? zc[8 + c] : 0.0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        a[c] += v * (C * zc[c] + Sn * zs[c]);
        if (grad) {
          const double rad = fr * (C * zc[c] + Sn * zs[c]);
          a[2 + c] += (rad * tx + v * m * (C0 * zc[c] + S0 * zs[c])) * S.iR0;
          a[4 + c] += (rad * ty + v * m * (C0 * zs[c] - S0 * zc[c])) * S.iR0;
          a[6 + c] += (rad * tz + fz * (C * zc[c] + Sn * zs[c])) * S.iR0;
        }
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) a[12 + c] += v * (C * zc[2 + c] + Sn * zs[2 + c]);
    }
  }
  __shared__ double sm[18][SMF_TH / 32];
#pragma unroll
  for (int c = 0; c < 18; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
    if ((tid & 31) == 0) sm[c][tid >> 5] = a[c];
  }
  __syncthreads();
  if (tid < 18) {
    double x = 0.0;
    for (int w = 0; w < SMF_TH / 32; ++w) x += sm[tid][w];
    if (tid >= 8 && tid < 12) x *= BEM_I_FP;  // F and dF carry 1/4pi
    out[18 * (size_t)ip + tid] = x;
  }
}

extern "C" int bem_launch_smfield(bem_smooth *F, const bem_dom_dev *D, const bem_qp *q, int grad, int type, int npts,
                                  const double *pts, const double *P, const double *dP, const double *pv,
                                  const double *dpv, double *out, int *again, unsigned *status, cudaStream_t st) {
  if (npts <= 0) return 0;
  if (launch_rest(F, q, 0, 1, status, st)) return -1;
  const sm_dev d = dev_view(F, D->ne, 0, true);
  if (launch_density(F, d, D, type, P, dP, pv, dpv, st)) return -1;
  k_sm_field<<<npts, SMF_TH, 0, st>>>(d, *D, grad, type, pts, P, dP, pv, dpv, out, again);
  bem_count_launches(1);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}
