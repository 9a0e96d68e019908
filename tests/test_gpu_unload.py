"""Calls on a context whose problem was unloaded and loaded again: the field sums'
order table and expansion, and the boundary sums' expansion, are given back with
the problem and made again.  Field calls of many points (images and expansion),
of points above the body beyond the expansion's reach (order table), boundary
values and the 9-point force, before and after, and on a smaller and a larger body in
between.

Tolerance: the same kernels on the same inputs, 1e-13 of the largest value of each
quantity (the geometric sum over a closed body cancels: it is left out)."""
import ctypes
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(g, api, ctx, prob, seed):
    """Solve prob and return its field sums, boundary values and force."""
    assert g.bemgpu_load(ctx, ctypes.byref(prob)) == 0, g.bemgpu_error(ctx)
    assert g.bemgpu_run(ctx) == 0, g.bemgpu_error(ctx)
    rng = np.random.default_rng(seed)
    res, launched = [], []
    for n, lo, hi, kind in ((4000, 0.36, 0.6, 1), (1500, 0.62, 0.75, 0x101)):
        r = rng.uniform(-0.35, 0.35, (n, 3))
        r[:, 2] = rng.uniform(lo, hi, n)
        out = np.zeros((n, 18))
        n0 = g.bemgpu_kernel_launches()
        assert g.bemgpu_field(ctx, 0, kind, n, api._p(r), api._p(out)) == 0, g.bemgpu_error(ctx)
        launched.append(g.bemgpu_kernel_launches() - n0)
        res += [out[:, :2], out[:, 2:8], out[:, 12:]]
    t = np.arange(8, dtype=np.int32)
    ze = rng.uniform(-0.8, 0.8, (8, 2))
    out = np.zeros((8, 9))
    assert g.bemgpu_boundary_field(ctx, 0, 1, 8, t.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), api._p(ze), api._p(out)) == 0
    F, N, rc = np.zeros(3), np.zeros(3), np.zeros(3)
    assert g.bemgpu_force(ctx, 1, api._p(rc), api._p(F), api._p(N)) == 0
    assert g.bemgpu_status(ctx) == 0
    return res + [out[:, :8], F], launched


def test_calls_after_unload_and_load():
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    vp, ip = ctypes.c_void_p, ctypes.POINTER(ctypes.c_int)
    g.bemgpu_load.argtypes = [vp, ctypes.POINTER(api.Problem)]
    g.bemgpu_unload.argtypes = [vp]
    g.bemgpu_field.argtypes = [vp] + [ctypes.c_int] * 3 + [api._d, api._d]
    g.bemgpu_boundary_field.argtypes = [vp, ctypes.c_int, ctypes.c_int, ctypes.c_int, ip, api._d, api._d]
    cases = [api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_ul_"), n=n, theta_deg=23.0, phi_deg=41.0,
                                                       lattice=((2.0, 0.0), (0.0, 2.0)), rot=((1.0, 2.0, 3.0), 37.0))) for n in (4, 2, 5)]
    probs = [c.problem() for c in cases]
    ctx, got = ctypes.c_void_p(), []
    assert g.bemgpu_create(0, None, ctypes.byref(ctx)) == 0
    try:
        for i in (0, 0, 1, 0, 2, 0):
            assert g.bemgpu_unload(ctx) == 0
            got.append((i,) + _calls(g, api, ctx, probs[i], 7))
        # an unloaded context refuses the calls
        assert g.bemgpu_unload(ctx) == 0
        x, y = np.array([[0.0, 0.0, 0.7]]), np.zeros((1, 18))
        assert g.bemgpu_field(ctx, 0, 1, 1, api._p(x), api._p(y)) == -2
    finally:
        g.bemgpu_destroy(ctx)
        for c, p in zip(cases, probs):
            c.free_problem(p)
            c.close()
    first = got[0]
    # both forms ran: images and expansion (eight launches), the order table (one)
    assert first[2][0] == 8 and first[2][1] == 1, first[2]
    for i, res, launched in got:
        if i == 0:
            assert launched == first[2]
            for x, y in zip(first[1], res):
                assert np.max(np.abs(x - y)) <= 1e-13 * np.max(np.abs(x))
