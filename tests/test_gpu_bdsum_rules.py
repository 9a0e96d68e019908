"""Boundary sums of the periodic domain from images and expansion on the rules that
test_gpu_bdsum.py leaves out: the 12 x 12 and 64 x 64 Gauss rules (triangles: 12 x 12 on
each of three parts), and on triangles the 4-point rule, whose centre point carries a
negative weight.  Against sums of lattice sums on the host as there, the target's own
element on its Duffy rule.

Tolerance (fixed before the first run): as there, 1e-10 of the largest sum on a turned
body, 1e-7 where mirrored triangles lie on the plane of the target."""
import ctypes

import numpy as np
import pytest

from test_gpu_bdsum import OBL, ROOT3, SQ, ZE_Q, ZE_T, _case, _duffy, _rw, _shape

pytestmark = pytest.mark.gpu


def _rule(tri, kind):
    if tri and kind == 0:
        z, e = np.array([-0.2, 0.4, -0.2, 0.0]), np.array([-ROOT3 / 5, 0.0, ROOT3 / 5, 0.0])
        return z, e, 0.5 * np.array([25.0, 25.0, 25.0, -27.0]) / 48.0
    x, w = np.polynomial.legendre.leggauss(12 if kind == 2 else 64)
    a, b = (v.ravel() for v in np.meshgrid(x, x, indexing="ij"))
    ww = np.outer(w, w).ravel()
    if not tri:
        return a, b, ww
    parts = [((3 + 2 * a + 2 * b + a * b) / 8, ROOT3 * (b - a) / 8),
             ((-3 + a - 5 * b - a * b) / 16, ROOT3 * (3 + 3 * a + b + a * b) / 16),
             ((-3 - 5 * a + b - a * b) / 16, ROOT3 * (-3 - a - 3 * b - a * b) / 16)]
    return (np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]),
            np.tile(ww * (1 + a / 4 + b / 4) / 24, 3))


@pytest.mark.parametrize("mesh,size,radius,lat,a,turned,kind", [
    ("quad", 1, 0.25, SQ, 0.8, True, 2), ("quad", 1, 0.25, SQ, 0.8, True, 3), ("quad", 2, 0.3, OBL, 1.2, True, 2),
    ("tri", 0, 0.28, OBL, 0.9, False, 0), ("tri", 1, 0.28, SQ, 0.8, False, 0), ("tri", 0, 0.28, OBL, 0.9, False, 2)])
def test_rules_match_lattice_sums(mesh, size, radius, lat, a, turned, kind):
    from bem3_aw_qd2_b200 import api
    g = api.libs()[1]
    case = _case(mesh, size, radius, 1.0, lat, a, turned)
    pr = case.problem()
    tri, Ne = mesh == "tri", pr.Ne
    view = lambda p, n, t=ctypes.c_double: np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(t)), (n,)).copy()
    ne = view(pr.dom_ne, 1, ctypes.c_int)[0]
    cr, cw = view(pr.cr, 12 * Ne).reshape(Ne, 3, 4), view(pr.cw, 9 * Ne).reshape(Ne, 3, 3)
    sid = np.abs(view(pr.sid, ne, ctypes.c_int)) - 1
    qp = np.array(list(pr.qp))
    val = np.concatenate([v.reshape(ne, 4, -1) for v in case.solution(0, ne)], axis=2)  # P, dP, pv, dpv
    P, dP = val[:, :, [0, 2, 3, 4]], val[:, :, [1, 5, 6, 7]]

    def terms(s, z, e, w, rt):  # (R, W w) of an element's points and its node functions there
        r, W = _rw(tri, cr[sid[s]], cw[sid[s]], z, e)
        return r - rt[:, None], W * w, np.sign(w), _shape(tri, z, e)

    ti_, ze = [], []
    for t in np.unique(np.linspace(0, ne - 1, 2).astype(int)):
        for x in (ZE_T if tri else ZE_Q)[:2]:
            ti_.append(t)
            ze.append(x)
    ti, ze = np.array(ti_, np.int32), np.array(ze, np.float64)
    rule, ref = _rule(tri, kind), np.zeros((len(ti), 4), np.complex128)
    for i, (t, (zt, et)) in enumerate(zip(ti, ze)):
        rt = _rw(tri, cr[sid[t]], cw[sid[t]], np.array([zt]), np.array([et]))[0][:, 0]
        els = [(t, terms(t, *_duffy(tri, zt, et), rt))] + [(s, terms(s, *rule, rt)) for s in range(ne) if s != t]
        G, dG, ret = api.qpgf(qp, np.concatenate([x[0] for _, x in els], axis=1).T)
        assert np.all(ret > 0)
        o = 0
        for s, (R, W, sg, N) in els:
            n, m = R.shape[1], len(N)
            gn = N @ (sg * np.linalg.norm(W, axis=0) * G[o:o + n])
            hn = N @ np.sum(dG[o:o + n].T * W, axis=0)
            ref[i] += gn @ dP[s, :m] - hn @ P[s, :m]
            o += n
    out = np.zeros((len(ti), 9))
    g.bemgpu_boundary_field.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                        ctypes.POINTER(ctypes.c_int), api._d, api._d]
    n0 = g.bemgpu_kernel_launches()
    assert g.bemgpu_boundary_field(case.ctx, 0, kind, len(ti), ti.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), api._p(ze),
                                   api._p(out)) == 0
    assert g.bemgpu_kernel_launches() - n0 >= 4  # the densities and the sums of the split
    got = out[:, :8].view(np.complex128)
    case.free_problem(pr)
    case.close()
    for c in (slice(0, 1), slice(1, 4)):  # potential, velocity
        err = np.max(np.abs(got[:, c] - ref[:, c])) / np.max(np.abs(ref[:, c]))
        assert err < (1e-10 if turned else 1e-7), err
