"""Field sums of many points from images and expansion (bemgpu_field's split, on a
plan whose ball holds the points) against the same points one call at a time (a
single point keeps its lattice sums): points near the body and far from it, one
far outlier that the ball leaves out, points level with nodes of the mesh (on
the lattice plane through a source: those points keep the lattice sums), quads
and triangles, square, triangular, oblique and sparse lattices, with and without
second derivatives.

Tolerance (fixed before the first run): lattice sums and split both carry a pair to
1e-13 of the sum's scale, second derivatives lose another 10: 1e-11 of the
largest value of each quantity, and 1e-7 at points level with a node, where the
lattice sums stop on rounding."""
import ctypes
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SQ = ((1.0, 0.0), (0.0, 1.0))
TRI = ((1.0, 0.0), (0.5, 0.75 ** 0.5))
OBL = ((1.0, 0.0), (0.3, 0.9))


@pytest.mark.parametrize("mesh,size,radius,lat,a,turned", [
    ("quad", 4, 0.3, SQ, 0.8, True), ("quad", 4, 0.3, SQ, 0.8, False), ("quad", 3, 0.35, OBL, 3.3, True),
    ("tri", 2, 0.25, TRI, 0.9, False)])
@pytest.mark.parametrize("kind", [0, 1, 0x100, 0x101])
def test_split_matches_single_points(mesh, size, radius, lat, a, turned, kind):
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    kw = dict(ico=size) if mesh == "tri" else dict(n=size)
    if turned:
        kw["rot"] = ((1.0, 2.0, 3.0), 37.0)
    case = api.Case.from_files(*meshgen.write_inputs(
        tempfile.mkdtemp(prefix="bem_fs_"), semi_axes=(radius,) * 3, lattice=tuple(tuple(a * x for x in v) for v in lat),
        theta_deg=23.0, phi_deg=41.0, **kw))
    case.solve()
    pr = case.problem()
    ren = np.ctypeslib.as_array(ctypes.cast(pr.ren, ctypes.POINTER(ctypes.c_double)), (12 * pr.Ne,)).reshape(-1, 4, 3).copy()
    case.free_problem(pr)
    g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
    rng = np.random.default_rng(11)
    n = 6000
    v = rng.standard_normal((n, 3))
    r = v / np.linalg.norm(v, axis=1, keepdims=True) * (radius * rng.uniform(1.08, 2.6, (n, 1)))
    r[17] = (0.1, -0.2, 9.0)  # far above
    r[30:60, 2] = ren[:30, 0, 2]  # level with a node
    r[30:60, 0] += radius
    out = np.zeros((n, 18))
    assert g.bemgpu_field(case.ctx, 0, kind, n, api._p(r), api._p(out)) == 0
    some = np.concatenate([np.arange(17, 40), np.arange(60, n, 331)])
    one = np.zeros((len(some), 18))
    for i, p in enumerate(some):
        x, y = np.ascontiguousarray(r[p]), np.zeros(18)
        assert g.bemgpu_field(case.ctx, 0, kind, 1, api._p(x), api._p(y)) == 0
        one[i] = y
    case.close()
    tol = np.where((some >= 30) & (some < 60), 1e-7, 1e-11)
    for c in (slice(0, 2), slice(2, 8), slice(8, 9), slice(9, 12), slice(12, 18)):
        err = np.max(np.abs(out[some][:, c] - one[:, c]), axis=1)
        assert np.all(err <= tol * np.max(np.abs(one[:, c]))), (c, np.max(err / tol))
