"""Two host threads with a context each on one GPU, on bodies whose expansions have
different degrees (their kernels differ in the shared memory that they take): each
loads, solves, takes the 9-point force and a field grid in a loop, and every call of
each thread succeeds with the values that the body gives alone.

Tolerance: the same kernels on the same inputs, 1e-13 of the largest value."""
import ctypes
import tempfile
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROUNDS = 40


def _work(g, api, ctx, prob, r):
    for call in (lambda: g.bemgpu_load(ctx, ctypes.byref(prob)), lambda: g.bemgpu_run(ctx)):
        if call() != 0:
            raise RuntimeError(g.bemgpu_error(ctx).decode())
    F, N, rc = np.zeros(3), np.zeros(3), np.zeros(3)
    out = np.zeros((len(r), 18))
    if g.bemgpu_force(ctx, 1, api._p(rc), api._p(F), api._p(N)) or \
            g.bemgpu_field(ctx, 0, 1, len(r), api._p(r), api._p(out)) or g.bemgpu_status(ctx):
        raise RuntimeError(g.bemgpu_error(ctx).decode())
    return [F, out[:, :2], out[:, 2:8], out[:, 12:]]


def test_threads_with_bodies_of_different_degrees():
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    g.bemgpu_load.argtypes = [ctypes.c_void_p, ctypes.POINTER(api.Problem)]
    g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
    # kR0 1 in a wide cell, and a body that nearly fills a small one: degrees far apart
    bodies = [dict(n=2, semi_axes=(0.16,) * 3, lattice=((1.6, 0.0), (0.0, 1.6))),
              dict(n=2, semi_axes=(0.28, 0.28, 0.5), lattice=((0.7, 0.0), (0.0, 0.7)))]
    cases = [api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_td_"), theta_deg=23.0, phi_deg=41.0,
                                                       rot=((1.0, 2.0, 3.0), 37.0), **b)) for b in bodies]
    probs = [c.problem() for c in cases]
    rng = np.random.default_rng(3)
    v = rng.standard_normal((4000, 3))
    grids = [v / np.linalg.norm(v, axis=1, keepdims=True) * (a * rng.uniform(1.1, 1.6, (4000, 1))) for a in (0.16, 0.5)]
    ctx = [ctypes.c_void_p(), ctypes.c_void_p()]
    bad = []

    def loop(i, ref):
        try:
            for _ in range(ROUNDS):
                for x, y in zip(_work(g, api, ctx[i], probs[i], grids[i]), ref):
                    if not np.max(np.abs(x - y)) <= 1e-13 * np.max(np.abs(y)):
                        raise RuntimeError("other values")
        except Exception as e:  # noqa: BLE001
            bad.append((i, str(e)))

    try:
        for c in ctx:
            assert g.bemgpu_create(0, None, ctypes.byref(c)) == 0
        refs = [_work(g, api, ctx[i], probs[i], grids[i]) for i in (0, 1)]
        th = [threading.Thread(target=loop, args=(i, refs[i])) for i in (0, 1)]
        for t in th:
            t.start()
        for t in th:
            t.join()
    finally:
        for c in ctx:
            if c:
                g.bemgpu_destroy(c)
        for c, p in zip(cases, probs):
            c.free_problem(p)
            c.close()
    assert not bad, bad
