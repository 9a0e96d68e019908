"""Boundary sums of the periodic domain (bemgpu_boundary_field, domain 0) from
images and expansion, against sums of lattice sums (bemgpu_qpgf) on the host:
every other element on the 4- or 9-point (triangles: 4- or 7-point) rule, the
target's own element on a Duffy rule around the target (24 x 160 points in each
of the triangles between the target and an edge).  Bodies as they stand (points
on the lattice plane through the target) and turned, quads and triangles,
square, triangular and oblique lattices; targets inside elements, near an edge
and on nodes of the 9-point rule.

Tolerance (fixed before the first run): the sums agree to the lattice sums' 1e-13
at each point; the own element's rules (polar with 12 points in radius, Duffy
with 24 x 160) converge to 1e-11 or better for targets this far from the edges; 1e-10
of the largest sum, and 1e-7 where mirrored elements lie on the plane of the
target (the lattice sums there stop on rounding, and both sides round apart)."""
import ctypes
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SQ = ((1.0, 0.0), (0.0, 1.0))
TRI = ((1.0, 0.0), (0.5, 0.75 ** 0.5))
OBL = ((1.0, 0.0), (0.3, 0.9))
CASES = [  # mesh, size, radius, stretch, lattice, period, turned
    ("quad", 1, 0.2, 1.0, SQ, 0.8, True),
    ("quad", 3, 0.3, 1.0, SQ, 0.8, False),
    ("quad", 4, 0.31, 1.35, TRI, 0.72, True),
    ("quad", 3, 0.35, 1.0, OBL, 3.3, True),
    ("tri", 1, 0.28, 1.0, OBL, 0.9, False),
    ("tri", 2, 0.3, 1.0, TRI, 0.8, False),
]
ZE_Q = [(0.2, -0.3), (-0.85, 0.6), (0.7745966692414834, 0.0)]
ZE_T = [(0.1, 0.05), (-0.2, 0.3), (0.0, 0.0)]
ROOT3 = 3.0 ** 0.5


def _case(mesh, size, radius, stretch, lat, a, turned):
    from bem3_aw_qd2_b200 import api, meshgen
    api.libs()[0].aqd2_set_verbose(0)
    kw = dict(ico=size) if mesh == "tri" else dict(n=size)
    if turned:
        kw["rot"] = ((1.0, 2.0, 3.0), 37.0)
    d = tempfile.mkdtemp(prefix="bem_bdsum_")
    c = api.Case.from_files(*meshgen.write_inputs(d, semi_axes=(radius, radius, radius * stretch), theta_deg=23.0,
                                                  lattice=tuple(tuple(a * x for x in v) for v in lat), phi_deg=41.0, **kw))
    c.solve()
    return c


def _shape(tri, z, e):
    """The node functions: nodes at +-1/sqrt3, of a triangle at (-1/5, -sqrt3/5), (2/5, 0), (-1/5, sqrt3/5)."""
    if tri:
        return np.array([1.0 - 2.5 * (z + ROOT3 * e), 1.0 + 5.0 * z, 1.0 - 2.5 * (z - ROOT3 * e)]) / 3.0
    z, e = ROOT3 * z, ROOT3 * e
    return 0.25 * np.array([(1 - z) * (1 - e), (1 + z) * (1 - e), (1 + z) * (1 + e), (1 - z) * (1 + e)])


def _rw(tri, cr, cw, z, e):
    """Position and Jacobian vector (quads: per d(zeta) d(eta); triangles: cw0, twice the area)."""
    r = cr[:, 0][:, None] + cr[:, 1][:, None] * z + cr[:, 2][:, None] * e
    if tri:
        return r, np.repeat(cw[:, 0][:, None], len(z), 1)
    return (r + cr[:, 3][:, None] * (z * e), cw[:, 0][:, None] + cw[:, 1][:, None] * z + cw[:, 2][:, None] * e)


def _rule(tri, kind):
    if tri and kind == 1:
        n0, n1, n2, n3 = 0.3480702390148154917985, 0.2052130961576726346557, 0.6028753385763033130539, 0.3554395089236065568357
        v0, v1 = 0.1259391805448271525957, 0.1323941527885061807376
        return (np.array([-n0, 2 * n0, -n0, n1, -2 * n1, n1, 0.0]), np.array([-n2, 0, n2, n3, 0, -n3, 0.0]),
                0.5 * np.array([v0] * 3 + [v1] * 3 + [0.225]))
    n = 2 if kind == 0 else 3
    x, w = np.polynomial.legendre.leggauss(n)
    z, e = (v.ravel() for v in np.meshgrid(x, x, indexing="ij"))
    return z, e, np.outer(w, w).ravel()


def _duffy(tri, zt, et):
    c = [(1.0, 0.0), (-0.5, ROOT3 / 2), (-0.5, -ROOT3 / 2)] if tri else [(-1.0, -1.0), (1.0, -1.0), (1.0, 1.0), (-1.0, 1.0)]
    # along the edge the integrand's nearest pole is the target's distance from the
    # edge (0.15 of half its length): a factor 1.16 a point and two, hence 160
    (x, w), (y, wy) = np.polynomial.legendre.leggauss(24), np.polynomial.legendre.leggauss(160)
    u, v = (a.ravel() for a in np.meshgrid(0.5 * (x + 1), 0.5 * (y + 1), indexing="ij"))
    wt = np.outer(0.5 * w, 0.5 * wy).ravel()
    Z, E, Wt = [], [], []
    for i in range(len(c)):
        (az, ae), (bz, be) = c[i], c[(i + 1) % len(c)]
        dz, de = az - zt + v * (bz - az), ae - et + v * (be - ae)
        Z.append(zt + u * dz)
        E.append(et + u * de)
        Wt.append(wt * u * abs((az - zt) * (be - ae) - (ae - et) * (bz - az)))
    # a triangle's (zeta, eta) area is 3 sqrt3 / 4 and cw0 is twice its area
    return np.concatenate(Z), np.concatenate(E), np.concatenate(Wt) * (2.0 / (3.0 * ROOT3) if tri else 1.0)


@pytest.mark.parametrize("mesh,size,radius,stretch,lat,a,turned", CASES)
@pytest.mark.parametrize("kind", [0, 1])
def test_boundary_sums_match_lattice_sums(mesh, size, radius, stretch, lat, a, turned, kind):
    from bem3_aw_qd2_b200 import api
    g = api.libs()[1]
    case = _case(mesh, size, radius, stretch, lat, a, turned)
    pr = case.problem()
    tri = mesh == "tri"
    if tri and kind == 0:
        kind = 1  # the nodes' rule is the quads'; triangles take the 7-point rule twice over
    Ne = pr.Ne
    view = lambda p, n, t=ctypes.c_double: np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(t)), (n,)).copy()
    ne = view(pr.dom_ne, 1, ctypes.c_int)[0]
    cr, cw = view(pr.cr, 12 * Ne).reshape(Ne, 3, 4), view(pr.cw, 9 * Ne).reshape(Ne, 3, 3)
    sid = np.abs(view(pr.sid, ne, ctypes.c_int)) - 1
    qp = np.array(list(pr.qp))
    val = np.concatenate([v.reshape(ne, 4, -1) for v in case.solution(0, ne)], axis=2)  # P, dP, pv, dpv
    P, dP = val[:, :, [0, 2, 3, 4]], val[:, :, [1, 5, 6, 7]]

    def green(R):
        n = R.shape[1]
        r = np.ascontiguousarray(R.T)
        G, dG, ret = np.zeros(n, np.complex128), np.zeros((n, 3), np.complex128), np.zeros(n, np.int32)
        assert g.bemgpu_qpgf(api._p(qp), api._p(r), n, api._p(G.view(np.float64)), api._p(dG.view(np.float64)),
                             ret.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
        assert np.all(ret > 0)
        return G, dG.T

    def sums(s, z, e, w, rt):
        r, W = _rw(tri, cr[sid[s]], cw[sid[s]], z, e)
        G, dG = green(r - rt[:, None])
        N = _shape(tri, z, e)
        m = len(N)
        gn = N @ (w * np.linalg.norm(W, axis=0) * G)
        hn = N @ (w * np.sum(dG * W, axis=0))
        return gn @ dP[s, :m] - hn @ P[s, :m]

    g.bemgpu_qpgf.argtypes = [api._d, api._d, ctypes.c_int, api._d, api._d, ctypes.POINTER(ctypes.c_int)]
    g.bemgpu_boundary_field.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                        ctypes.POINTER(ctypes.c_int), api._d, api._d]
    els = np.unique(np.linspace(0, ne - 1, 4).astype(int))
    tgt = [(t, ze) for t in els for ze in (ZE_T if tri else ZE_Q)]
    ti = np.array([t for t, _ in tgt], np.int32)
    ze = np.array([x for _, x in tgt], np.float64)
    out = np.zeros((len(tgt), 9))
    rule = _rule(tri, kind)
    ref = np.zeros((len(tgt), 4), np.complex128)
    for i, (t, (zt, et)) in enumerate(tgt):
        rt = _rw(tri, cr[sid[t]], cw[sid[t]], np.array([zt]), np.array([et]))[0][:, 0]
        ref[i] = sums(t, *_duffy(tri, zt, et), rt) + sum(sums(s, *rule, rt) for s in range(ne) if s != t)
    assert g.bemgpu_boundary_field(case.ctx, 0, kind, len(tgt), ti.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), api._p(ze),
                                   api._p(out)) == 0
    got = out[:, :8].view(np.complex128)
    case.free_problem(pr)
    case.close()
    for c in (slice(0, 1), slice(1, 4)):  # potential, velocity
        err = np.max(np.abs(got[:, c] - ref[:, c])) / np.max(np.abs(ref[:, c]))
        assert err < (1e-10 if turned else 1e-7), err
