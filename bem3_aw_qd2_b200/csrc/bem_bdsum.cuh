// Boundary sums of the periodic domain (k_bdval, bem_post.cuh) with the images
// and the expansion of bem_smooth.cu; included at its end.
//
// A target sums the Green's function over every element's rule points and over
// the polar rule of its own element: (9 ne + 6144) lattice sums for the 9-point
// force at each of 9 ne points.  Here the images are closed forms; the rest of
// every point is contracted once with the boundary values into K coefficients
// (k_sm_density, k_sm_density_T) that a target meets with its own K functions;
// and where a single point's rest is needed (the target's own element, whose
// rule points the polar rule replaces, and points on the lattice plane through
// the target, where the reference's sums stop on rounding and are kept), it
// comes from the expansion about the target (sm_rest).  A 9-point force of 150
// turned quads takes 0.98 ms for 19.9 of k_bdval, 0.89 of it k_sm_bdsum.  A target
// with a quarter of its points on its plane (flat bodies across z) keeps the
// lattice sums: there they are the cheaper form.
#pragma once

#define SMD_NCH 32     // chunks of elements a density is summed in
#define SMD_TH 160
#define SMB_TH 128
#define SMB_CH 64

// Z[chunk][lm][2 c + part]: sum over the chunk's elements and rule points of
// w (|W| phi D_c - W . grad phi S_c), with (D, S)_c the normal derivative and
// the value of the potential (c = 0) and of the velocity components (c = 1 .. 3)
__global__ void __launch_bounds__(SMD_TH) k_sm_density(const __grid_constant__ sm_dev S, bem_dom_dev D, int type,
                                                       const double *__restrict__ P, const double *__restrict__ dP,
                                                       const double *__restrict__ pv, const double *__restrict__ dpv) {
  extern __shared__ double sm_raw[];
  const int ch = blockIdx.x, m = blockIdx.y, tid = threadIdx.x;
  const int nl = S.lmax + 1 - m, nf = m ? 2 : 1, nout = nl * 2 * nf;
  double *den = sm_raw;                     // [16][SMV_PT]: D (re, im) x 4, then -S
  double *val = den + 16 * SMV_PT;          // [nl][2 nf][SMV_PT]
  double acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = 0.0;
  // the chunk's rule points, SMV_PT at a time
  const int nr = D.has_tri ? max(rule_points(type), tri_rule_points(type)) : rule_points(type);
  const long long npts = (long long)((D.ne - ch + SMD_NCH - 1) / SMD_NCH) * nr;
  for (long long p0 = 0; p0 < npts; p0 += SMV_PT) {
    const int np = (int)min((long long)SMV_PT, npts - p0);
    __syncthreads();
    if (tid < np) {
      const int s = ch + SMD_NCH * (int)((p0 + tid) / nr), i = (int)((p0 + tid) % nr);
      const int se = abs(D.sid[s]) - 1;
      const bool tri = D.has_tri && D.npe[se] == 3, is = i < (tri ? tri_rule_points(type) : rule_points(type));
      double z, e, w, r[3], W[3];
      bd_source_point(D, se, tri, type, is ? i : 0, z, e, w, r, W);
      if (!is) w = 0.0;
      cplx Pn, dPn, pvn[3], dpvn[3];
      interp_bv(type, is ? i : 0, z, e, s, P, dP, pv, dpv, Pn, dPn, pvn, dpvn, tri);
      den[0 * SMV_PT + tid] = w * dPn.re;
      den[1 * SMV_PT + tid] = w * dPn.im;
      den[8 * SMV_PT + tid] = -w * Pn.re;
      den[9 * SMV_PT + tid] = -w * Pn.im;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        den[(2 + 2 * c) * SMV_PT + tid] = w * dpvn[c].re;
        den[(3 + 2 * c) * SMV_PT + tid] = w * dpvn[c].im;
        den[(10 + 2 * c) * SMV_PT + tid] = -w * pvn[c].re;
        den[(11 + 2 * c) * SMV_PT + tid] = -w * pvn[c].im;
      }
      sm_point_values(S, m, nf, r, W, val + tid);
    }
    __syncthreads();
    if (tid < nout) {
      const double *v = val + (size_t)tid * SMV_PT, *d = den + (tid & 1 ? 8 * SMV_PT : 0);
      const int q0 = tid % np;
      for (int q = 0; q < np; ++q) {
        const int qq = q + q0 < np ? q + q0 : q + q0 - np;
        const double x = v[qq];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = fma(x, d[c * SMV_PT + qq], acc[c]);
      }
    }
  }
  // the value's and the derivative's thread are neighbours
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], 1);
  if (tid < nout && !(tid & 1)) {
    const int l = m + tid / (2 * nf), sine = (tid % (2 * nf)) >> 1;
    double *o = S.Z + ((size_t)ch * S.Kp + sm_idx(l, m, sine)) * 8;
#pragma unroll
    for (int c = 0; c < 8; ++c) o[c] = acc[c];
  }
}

// the chunks summed, into the first
__global__ void __launch_bounds__(SMB_TH) k_sm_density_sum(const __grid_constant__ sm_dev S) {
  const int i = blockIdx.x * SMB_TH + threadIdx.x;
  if (i >= 8 * S.K) return;
  double x = 0.0;
#pragma unroll
  for (int ch = 0; ch < SMD_NCH; ++ch) x += S.Z[(size_t)ch * 8 * S.Kp + i];
  S.Z[i] = x;
}
// Zt[l'm'][c] = sum_lm T_lm,l'm' Z[lm][c]: a block per l'm', the lm over its threads
__global__ void __launch_bounds__(SMB_TH) k_sm_density_T(const __grid_constant__ sm_dev S) {
  const int c0 = blockIdx.x;
  const double *T = S.T + (size_t)c0 * 2 * S.Kp;
  double a[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) a[c] = 0.0;
  for (int r = threadIdx.x; r < S.K; r += SMB_TH) {
    const double *z = S.Z + 8 * r;
    const double tr = T[r], ti = T[S.Kp + r];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[2 * c] += tr * z[2 * c] - ti * z[2 * c + 1];
      a[2 * c + 1] += tr * z[2 * c + 1] + ti * z[2 * c];
    }
  }
  __shared__ double sm[8][SMB_TH / 32];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
    if ((threadIdx.x & 31) == 0) sm[c][threadIdx.x >> 5] = a[c];
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double x = 0.0;
    for (int w = 0; w < SMB_TH / 32; ++w) x += sm[threadIdx.x][w];
    S.Zt[8 * c0 + threadIdx.x] = x;
  }
}

// degree that G_s needs at |R|: tabled in steps of 2 R0 / 8
__device__ __forceinline__ int sm_degree(const sm_dev &S, const double R[3]) {
  return S.lcut[min(7, (int)(8.0 * sqrt(dot3(R, R)) / S.rho))];
}
// Orders m0, m0 + step, ... of G_s(R) and its gradient, from the expansion about
// R = 0 (|R| <= 2 R0) to degree L; cg[l]: 1 / ((2 l + 1) (2 l + 3))
__device__ __noinline__ void sm_rest(const sm_dev &S, const double *cg, double rx, double ry, double rz, int L, int m0,
                                     int step, bem_gval &o) {
  const double ir = 1.0 / S.rho, x = rx * ir, y = ry * ir, z = rz * ir, s2 = x * x + y * y + z * z;
  const double kk2 = S.k * S.k * S.rho * S.rho, z2 = kk2 * s2;
  double g[2 * BEM_SM_MAXL + 2];  // g_0 .. g_{L + 1}, downward from the series of the two above
  {
    double u[2];
    for (int w = 0; w < 2; ++w) {
      const double l2 = 2.0 * (L + 2 - w) + 1.0;
      double t = 1.0, s = 1.0;
      for (int n = 1; n < 100; ++n) {
        t *= -0.5 * z2 / (n * (l2 + 2.0 * n));
        s += t;
        if (fabs(t) < 1e-18 * fabs(s)) break;
      }
      u[w] = s;
    }
    double up = u[0], at = u[1];
    g[L + 1] = at;
    for (int l = L + 1; l > 0; --l) {
      const double c = at - z2 * cg[l] * up;
      up = at;
      at = c;
      g[l - 1] = c;
    }
  }
  cplx v = cmk(0, 0), gx = v, gy = v, gz = v;
  double C = 1.0, Sn = 0.0, C0 = 0.0, S0 = 0.0;
  int at = 0;
  for (int m = m0; m <= L; m += step) {
    for (; at < m; ++at) {
      C0 = C;
      S0 = Sn;
      const double c2 = C * x - Sn * y;
      Sn = C * y + Sn * x;
      C = c2;
    }
    double t1 = S.rec[m * (m + 1) + 2 * m], t0 = 0.0, p1 = 0.0, p0 = 0.0, q1 = 0.0, q0 = 0.0;
    // sums over l of (sigma_lm + sigma_l-m) and i (sigma_lm - sigma_l-m) times
    // g Theta, its factor of the gradient along z and its radial factor
    cplx a = cmk(0, 0), b = a, az = a, bz = a, ar = a, br = a;
    for (int l = m; l <= L; ++l) {
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
      const double2 sp = reinterpret_cast<const double2 *>(S.sig)[l * l + l + m];
      const double2 sn = reinterpret_cast<const double2 *>(S.sig)[l * l + l - m];
      const double f = m ? 1.0 : 0.5;  // m = 0: one function
      const cplx A = cmk(f * (sp.x + sn.x), f * (sp.y + sn.y)), B = cmk(sn.y - sp.y, sp.x - sn.x);
      const double gt = g[l] * t1, fz = g[l] * p1, fr = 2.0 * g[l] * q1 - kk2 * g[l + 1] / (2.0 * l + 3.0) * t1;
      a = cadd(a, cscale(A, gt));
      b = cadd(b, cscale(B, gt));
      az = cadd(az, cscale(A, fz));
      bz = cadd(bz, cscale(B, fz));
      ar = cadd(ar, cscale(A, fr));
      br = cadd(br, cscale(B, fr));
    }
    v = cadd(v, cadd(cscale(a, C), cscale(b, Sn)));
    const cplx rad = cadd(cscale(ar, C), cscale(br, Sn)), zz = cadd(cscale(az, C), cscale(bz, Sn));
    gx = cadd(gx, cadd(cscale(rad, x), cscale(cadd(cscale(a, C0), cscale(b, S0)), (double)m)));
    gy = cadd(gy, cadd(cscale(rad, y), cscale(csub(cscale(b, C0), cscale(a, S0)), (double)m)));
    gz = cadd(gz, cadd(cscale(rad, z), zz));
  }
  o.g = v;
  o.gx = cscale(gx, ir);
  o.gy = cscale(gy, ir);
  o.gz = cscale(gz, ir);
}

// images m0 .. nimg - 1 of G and its gradient at R
__device__ __forceinline__ void sm_images_at(const sm_dev &S, const double *im, int m0, const double R[3], bem_gval &o) {
  const double kpi = S.k * 0.31830988618379067154, rz2 = R[2] * R[2];
  cplx g = cmk(0, 0), gx = g, gy = g, gz = g;
  for (int m = m0; m < S.nimg; ++m) {
    const double px = R[0] + im[3 * m], py = R[1] + im[3 * m + 1];
    double a, c, fr, fi;
    sm_image(kpi, S.k, px, py, rz2, im[3 * m + 2], a, c, fr, fi);
    g = cadd(g, cmk(a, c));
    gx = cadd(gx, cmk(fr * px, fi * px));
    gy = cadd(gy, cmk(fr * py, fi * py));
    gz = cadd(gz, cmk(fr * R[2], fi * R[2]));
  }
  o.g = cscale(g, BEM_I_FP);
  o.gx = cscale(gx, BEM_I_FP);
  o.gy = cscale(gy, BEM_I_FP);
  o.gz = cscale(gz, BEM_I_FP);
}

// a[0 .. 7] += w (|W| G (dP, dpv) - W . grad G (P, pv))
__device__ __forceinline__ void bd_add(double (&a)[9], const bem_gval &gv, const double W[3], double w, const cplx &Pn,
                                       const cplx &dPn, const cplx pvn[3], const cplx dpvn[3]) {
  const cplx G = cscale(gv.g, w * sqrt(W[0] * W[0] + W[1] * W[1] + W[2] * W[2]));
  const cplx H = cscale(cadd(cadd(cscale(gv.gx, W[0]), cscale(gv.gy, W[1])), cscale(gv.gz, W[2])), w);
  const cplx t0 = csub(cmul(G, dPn), cmul(H, Pn));
  a[0] += t0.re;
  a[1] += t0.im;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const cplx t = csub(cmul(G, dpvn[j]), cmul(H, pvn[j]));
    a[2 + 2 * j] += t.re;
    a[3 + 2 * j] += t.im;
  }
}

__device__ __forceinline__ void bd_sub(bem_gval &a, const bem_gval &b) {
  a.g = csub(a.g, b.g);
  a.gx = csub(a.gx, b.gx);
  a.gy = csub(a.gy, b.gy);
  a.gz = csub(a.gz, b.gz);
}

static __device__ __noinline__ unsigned sm_lattice(const bem_qp &q, double x, double y, double z, bem_gval &gv) {
  const int rc = bem_qpgf(q, x, y, z, gv);
  return rc >= 0 ? 0u : (rc == -12 || rc == -23) ? BEM_ST_RAYLEIGH : BEM_ST_QPGF_LIMIT;
}

// One block per target; out as k_bdval's.
//
// Bound by the latency of the points' rests: a block has some 60 of them (the
// target's element on the rest's rule, its own rule points, the points on its
// lattice plane), each a double loop over (l, m).  So the block lists them and
// takes SMB_CH at a time, a lane per point, the orders m dealt to the warps.
// The element's own points are summed against its four node functions, which
// meet the boundary values once at the end.  Three blocks an SM (168 registers, a
// few spills) keep 320 targets in one wave: the centres of 320 triangles 1.9 -> 1.5
// ms for two blocks of 255, nine points of 150 quads 0.98 ms with either.
__global__ void __launch_bounds__(SMB_TH, 3) k_sm_bdsum(const __grid_constant__ sm_dev S, bem_dom_dev D,
                                                     const __grid_constant__ bem_qp q, int type,
                                                     const int *__restrict__ tgt_t, const double *__restrict__ tgt_ze,
                                                     const double *__restrict__ P, const double *__restrict__ dP,
                                                     const double *__restrict__ pv, const double *__restrict__ dpv,
                                                     double *__restrict__ out, unsigned *status) {
  __shared__ double im[3 * BEM_SM_MAXIMG], gl[BEM_SM_MAXL + 2], cg[2 * BEM_SM_MAXL + 2];
  __shared__ polar_tab T;
  __shared__ int list[SMB_CH + SMB_TH], wcnt[SMB_TH / 32];
  __shared__ double sR[3][SMB_CH], part[SMB_TH / 32][8][SMB_CH];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int e = tid; e < 3 * S.nimg; e += SMB_TH) im[e] = S.img[e];
  for (int l = tid; l < 2 * BEM_SM_MAXL + 2; l += SMB_TH) cg[l] = 1.0 / ((2.0 * l + 1.0) * (2.0 * l + 3.0));
  const int ip = blockIdx.x, t = tgt_t[ip];
  const double zt = tgt_ze[2 * ip], et = tgt_ze[2 * ip + 1];
  const int te = abs(D.sid[t]) - 1;
  bem_el elt;
  bem_load_el(D.cr, D.cw, te, elt);
  double rt[3], wt_[3];
  bem_rw_ref(elt, zt, et, rt, wt_);
  const bool ttri = D.has_tri && D.npe[te] == 3;
  unsigned st = 0;
  {
    double r[5], th[5];
    if (ttri) bem_tri_node_r_th(zt, et, r, th);
    else bem_node_r_th(zt, et, r, th);
    polar_fill(T, r, th, ttri ? 384 : 512, st);
  }
  const double tx = (rt[0] - S.cx) * S.iR0, ty = (rt[1] - S.cy) * S.iR0, tz = (rt[2] - S.cz) * S.iR0;
  const double ts2 = tx * tx + ty * ty + tz * tz;
  if (tid == 0) sm_gl(S.lmax, S.kR0 * S.kR0 * ts2, gl, 1);
  const int nr = D.has_tri ? max(rule_points(type), tri_rule_points(type)) : rule_points(type);
  const int nit = D.ne * nr, npol = (ttri ? 384 : 512) * BEM_GLN;
  // the rest's rule on the target's element; an element across z has all its
  // points on the plane and is summed on the polar rule alone
  double dz = 0.0;
  for (int c = 1; c < (ttri ? 3 : 4); ++c) dz += fabs(elt.cr[2][c]);
  const bool flat = dz < BEM_FAR_PLANE_TOL;
  const double R2 = el_circum2(elt, ttri);
  const int tier = tier_image(S.cut * S.cut / R2, S.k * S.k * R2, ttri, ttri || quad_tier_shape(elt));
  const int nrest = D.far_rule && tier >= 0 ? BEM_TIER_N0 - tier : BEM_GLN;
  const int nres = flat ? 0 : rule_npts(nrest, ttri);

  // Points: rule point code, then the polar rule, then the rest's rule on the
  // target's element.  False where an element has fewer rule points.
  auto point = [&](int code, int &s, double &z, double &e, double &w, double vR[3], double vW[3], bool &stri) {
    if (code < nit) {
      s = code / nr;
      const int i = code % nr, se = abs(D.sid[s]) - 1;
      stri = D.has_tri && D.npe[se] == 3;
      if (i >= (stri ? tri_rule_points(type) : rule_points(type))) return false;
      bd_source_point(D, se, stri, type, i, z, e, w, vR, vW);
      for (int d = 0; d < 3; ++d) vR[d] = __dsub_rn(vR[d], rt[d]);
      return true;
    }
    s = t;
    stri = ttri;
    if (code < nit + npol) {
      const int idx = (code - nit) / BEM_GLN, ir = (code - nit) % BEM_GLN;
      const double rm = T.rm[idx], sth = T.s[idx], cth = T.c[idx];
      const double rr = 0.5 * rm * (c_q.xl[ir] + 1.0);
      w = T.w[idx] * 0.5 * rm * c_q.wl[ir] * rr;
      z = rr * cth + zt;
      e = rr * sth + et;
      double K[3];
      bem_K(elt, rr, cth, sth, zt, et, K);
      for (int d = 0; d < 3; ++d) {
        vR[d] = rr * K[d];
        vW[d] = ttri ? elt.cw[d][0] * (2.0 / (3.0 * BEM_SQ3)) : elt.cw[d][0] + elt.cw[d][1] * z + elt.cw[d][2] * e;
      }
    } else {
      rule_pt(nrest, ttri, code - nit - npol, z, e, w);
      bem_rw(elt, z, e, vR, vW);
      for (int d = 0; d < 3; ++d) vR[d] -= rt[d];
    }
    return true;
  };
  // points on the plane: where a quarter of all lie there, every point is a lattice sum
  int met = 0;
  for (int it = tid; it < nit; it += SMB_TH) {
    int s;
    double z, e, w, vR[3], vW[3];
    bool stri;
    if (point(it, s, z, e, w, vR, vW, stri)) met += fabs(vR[2]) < BEM_FAR_PLANE_TOL;
  }
  met = __reduce_add_sync(0xffffffffu, met);
  if (lane == 0) wcnt[wid] = met;
  __syncthreads();
  met = 0;
  for (int w = 0; w < SMB_TH / 32; ++w) met += wcnt[w];
  const bool sums = 4 * (long long)met > nit;

  double a[9], v[16];  // sums; G and H of the four node functions of the target's element
#pragma unroll
  for (int c = 0; c < 9; ++c) a[c] = 0.0;
#pragma unroll
  for (int c = 0; c < 16; ++c) v[c] = 0.0;
  auto add_own = [&](const bem_gval &gv, const double vW[3], double w, double z, double e) {
    double N[4];
    bem_Nn(ttri, z, e, N);
    const cplx G = cscale(gv.g, w * sqrt(dot3(vW, vW)));
    const cplx H = cscale(cadd(cadd(cscale(gv.gx, vW[0]), cscale(gv.gy, vW[1])), cscale(gv.gz, vW[2])), w);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      v[2 * n] += N[n] * G.re;
      v[2 * n + 1] += N[n] * G.im;
      v[8 + 2 * n] += N[n] * H.re;
      v[9 + 2 * n] += N[n] * H.im;
    }
  };
  auto add_source = [&](const bem_gval &gv, const double vW[3], double w, int s, int i, double z, double e, bool stri) {
    cplx Pn, dPn, pvn[3], dpvn[3];
    interp_bv(type, i, z, e, s, P, dP, pv, dpv, Pn, dPn, pvn, dpvn, stri);
    bd_add(a, gv, vW, w, Pn, dPn, pvn, dpvn);
  };
  // the listed points [n0, n0 + n)
  auto take = [&](int n0, int n) {
    int s = t, code = 0;
    double z = 0.0, e = 0.0, w = 0.0, vR[3] = {0, 0, 0}, vW[3] = {0, 0, 0};
    bool stri = false;
    if (tid < n) {
      code = list[n0 + tid];
      point(code, s, z, e, w, vR, vW, stri);
      for (int d = 0; d < 3; ++d) sR[d][tid] = vR[d];
    }
    __syncthreads();
    for (int p0 = 0; p0 < n; p0 += 32) {
      const int p = min(p0 + lane, n - 1);
      const double R[3] = {sR[0][p], sR[1][p], sR[2][p]};
      bem_gval g;
      sm_rest(S, cg, R[0], R[1], R[2], __reduce_max_sync(0xffffffffu, sm_degree(S, R)), wid, SMB_TH / 32, g);
      const double c[8] = {g.g.re, g.g.im, g.gx.re, g.gx.im, g.gy.re, g.gy.im, g.gz.re, g.gz.im};
      if (p0 + lane < n) {
#pragma unroll
        for (int j = 0; j < 8; ++j) part[wid][j][p] = c[j];
      }
    }
    __syncthreads();
    if (tid < n) {
      double c[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        c[j] = part[0][j][tid];
#pragma unroll
        for (int u = 1; u < SMB_TH / 32; ++u) c[j] += part[u][j][tid];
      }
      bem_gval g = {cmk(c[0], c[1]), cmk(c[2], c[3]), cmk(c[4], c[5]), cmk(c[6], c[7])};
      if (code < nit + npol) {
        bem_gval l = {};
        if (code >= nit || s != t) st |= sm_lattice(q, vR[0], vR[1], vR[2], l);
        bd_sub(l, g);
        g = l;
        if (code >= nit) {
          sm_images_at(S, im, 1, vR, l);
          bd_sub(g, l);
        }
      }
      if (code < nit) add_source(g, vW, w, s, code % nr, z, e, stri);
      else add_own(g, vW, w, z, e);
    }
    __syncthreads();
  };
  // the rest of every element's rule points: sum_k phi_k(target) Zt_k, a thread per order
  for (int m = sums ? S.lmax + 1 : tid; m <= S.lmax; m += SMB_TH) {
    double C = 1.0, Sn = 0.0;
    for (int b = 0; b < m; ++b) {
      const double c2 = C * tx - Sn * ty;
      Sn = C * ty + Sn * tx;
      C = c2;
    }
    if (m) { C *= 1.4142135623730950488; Sn *= 1.4142135623730950488; }
    double t1 = S.rec[m * (m + 1) + 2 * m], t0 = 0.0;
    for (int l = m; l <= S.lmax; ++l) {
      if (l > m) {
        const double *rr = S.rec + l * (l + 1) + 2 * m;
        const double t2 = rr[0] * (tz * t1 - rr[1] * ts2 * t0);
        t0 = t1;
        t1 = t2;
      }
      const double f = gl[l] * t1;
      const double *zc = S.Zt + 8 * sm_idx(l, m, 0);
#pragma unroll
      for (int c = 0; c < 8; ++c) a[c] += f * (C * zc[c] + (m ? Sn * zc[8 + c] : 0.0));
    }
  }
  // The other elements' points: images (or all of G) and the geometric sum.  The
  // element itself: the home image on the polar rule around (zt, et), the other
  // images on the 12 x 12 rule, the rest on its own; at a polar point on the plane
  // what the lattice sum has beyond these.
  int nlist = 0;
  const int ntot = nit + npol + nres;
  for (int c0 = 0; c0 < ntot || nlist; c0 += SMB_TH) {
    const int code = c0 + tid;
    int s = t;
    double z, e, w, vR[3], vW[3];
    bool stri, rest = false;
    if (code < ntot && point(code, s, z, e, w, vR, vW, stri)) {
      const bool on = fabs(vR[2]) < BEM_FAR_PLANE_TOL;
      bem_gval gv;
      if (code >= nit + npol) {
        rest = true;
      } else if (code >= nit) {
        if (flat) st |= sm_lattice(q, vR[0], vR[1], vR[2], gv);
        else if (on) rest = true;
        else bem_g0(S.k, vR, gv);
        if (!rest) add_own(gv, vW, w, z, e);
      } else if (s == t) {
        rest = !sums;
      } else {
        if (sums) st |= sm_lattice(q, vR[0], vR[1], vR[2], gv);
        else if (on) rest = true;
        else sm_images_at(S, im, 0, vR, gv);
        if (!rest) add_source(gv, vW, w, s, code % nr, z, e, stri);
        const double iR = 1.0 / sqrt(dot3(vR, vR));
        a[8] += (D.sid[s] < 0 ? -1.0 : 1.0) * w * dot3(vR, vW) * iR * iR * iR * BEM_I_FP;
      }
    }
    if (__syncthreads_or(rest)) {
      const unsigned who = __ballot_sync(0xffffffffu, rest);
      if (lane == 0) wcnt[wid] = __popc(who);
      __syncthreads();
      int at = nlist + __popc(who & ((1u << lane) - 1));
#pragma unroll
      for (int u = 0; u < SMB_TH / 32; ++u) {
        if (u < wid) at += wcnt[u];
        nlist += wcnt[u];
      }
      if (rest) list[at] = code;
      __syncthreads();
    }
    while (nlist >= SMB_CH || (nlist && c0 + SMB_TH >= ntot)) {
      const int n = min(nlist, SMB_CH);
      nlist -= n;
      take(nlist, n);
    }
  }
  for (int pt = tid; !flat && pt < rule_npts(BEM_GLN, ttri); pt += SMB_TH) {
    double z, e, w, vR[3], vW[3];
    rule_pt(BEM_GLN, ttri, pt, z, e, w);
    bem_rw(elt, z, e, vR, vW);
    for (int d = 0; d < 3; ++d) vR[d] -= rt[d];
    bem_gval gv;
    sm_images_at(S, im, 1, vR, gv);
    add_own(gv, vW, w, z, e);
  }
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const size_t o = (size_t)t * 4 + n;
    const cplx G = cmk(v[2 * n], v[2 * n + 1]), H = cmk(v[8 + 2 * n], v[9 + 2 * n]);
    const cplx t0 = csub(cmul(G, cmk(dP[2 * o], dP[2 * o + 1])), cmul(H, cmk(P[2 * o], P[2 * o + 1])));
    a[0] += t0.re;
    a[1] += t0.im;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const size_t oc = 2 * (3 * o + c);
      const cplx tc = csub(cmul(G, cmk(dpv[oc], dpv[oc + 1])), cmul(H, cmk(pv[oc], pv[oc + 1])));
      a[2 + 2 * c] += tc.re;
      a[3 + 2 * c] += tc.im;
    }
  }
  // the element's own F (geometric polar rule, zero for plane elements)
  const bool plane = D.plane[te] != 0;
  if (!plane) a[8] += (D.sid[t] < 0 ? -1.0 : 1.0) * polar_F_partial(elt, zt, et, st) * BEM_I_FP * bem_bdC(elt);
  set_status(status, st);
  __shared__ double sm[9][SMB_TH / 32];
#pragma unroll
  for (int c = 0; c < 9; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
    if ((threadIdx.x & 31) == 0) sm[c][threadIdx.x >> 5] = a[c];
  }
  __syncthreads();
  if (threadIdx.x < 9) {
    double x = 0.0;
    for (int w = 0; w < SMB_TH / 32; ++w) x += sm[threadIdx.x][w];
    out[9 * (size_t)ip + threadIdx.x] = x;
  }
}

// the densities of a rule's sources with the boundary values given
static int launch_density(const bem_smooth *S, const sm_dev &d, const bem_dom_dev *D, int type, const double *P,
                          const double *dP, const double *pv, const double *dpv, cudaStream_t st) {
  k_sm_density<<<dim3(SMD_NCH, S->lmax + 1), SMD_TH, sm_point_smem(16, S->lmax), st>>>(d, *D, type, P, dP, pv, dpv);
  k_sm_density_sum<<<(8 * S->K + SMB_TH - 1) / SMB_TH, SMB_TH, 0, st>>>(d);
  k_sm_density_T<<<S->K, SMB_TH, 0, st>>>(d);
  bem_count_launches(3);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int bem_launch_bdsum(bem_smooth *S, const bem_dom_dev *D, const bem_qp *q, int type, int ntgt, const int *tgt_t,
                                const double *tgt_ze, const double *P, const double *dP, const double *pv,
                                const double *dpv, double *out, unsigned *status, cudaStream_t st) {
  if (ntgt <= 0) return 0;
  if (!(S->have0 <= S->first && S->first < S->have1) && launch_rest(S, q, S->first, 1, status, st)) return -1;
  const sm_dev d = dev_view(S, D->ne, S->first, true);
  if (launch_density(S, d, D, type, P, dP, pv, dpv, st)) return -1;
  k_sm_bdsum<<<ntgt, SMB_TH, 0, st>>>(d, *D, *q, type, tgt_t, tgt_ze, P, dP, pv, dpv, out, status);
  bem_count_launches(1);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}
