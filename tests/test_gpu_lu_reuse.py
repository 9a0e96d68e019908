"""One bem_lu and one matrix buffer used for systems of different sizes in turn, on
both sides of the size up to which a factorisation is a kept graph (2048): a
larger system moves the row map and the tournament's scratch, whose addresses a
graph of an earlier, smaller one holds.  Both precisions, and the same through a
context that solves bodies of different sizes, with and without an unload between.

Tolerances: the residual relative to ||A|| ||X|| as test_gpu_lu.py holds it (1e-13
FP64, 2e-6 complex FP32); the context's solutions are those of the same kernels on
the same inputs, 1e-13 of the largest value (mixed precision, whose refinement ends
at that size of a correction: 1e-12)."""
import ctypes
import tempfile

import numpy as np
import pytest

from test_gpu_lu import random_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(300, 2337, 300), (2337, 300, 417, 300), (40, 300, 2500, 40, 300)])
@pytest.mark.parametrize("precision", ["z", "c"])
def test_sizes_in_turn(sizes, precision):
    import torch
    from bem3_aw_qd2_b200 import api
    _, g = api.libs()
    vp = ctypes.c_void_p
    factor, solve = getattr(g, "bem_lu_factor_" + precision), getattr(g, "bem_lu_solve_" + precision)
    g.bem_lu_init.argtypes = [vp, ctypes.c_int]
    g.bem_lu_free.argtypes = [vp]
    factor.argtypes = [vp, vp, ctypes.c_int, vp]
    solve.argtypes = [vp, vp, ctypes.c_int, ctypes.c_int, vp, vp]
    g.bem_lu_status.argtypes = [vp, vp]
    g.bem_lu_status.restype = ctypes.c_uint
    dt = np.complex128 if precision == "z" else np.complex64
    w = ctypes.create_string_buffer(4096)
    wp = ctypes.addressof(w)
    assert g.bem_lu_init(wp, 0) == 0
    res = []
    try:
        st = torch.cuda.Stream()
        Ad = torch.zeros(max(sizes) ** 2, dtype=torch.complex128 if precision == "z" else torch.complex64, device="cuda")
        for i, n in enumerate(sizes):
            A, B = random_system(n, 2, seed=90 + 7 * i + n, permuted=True)
            Ad[:n * n] = torch.from_numpy(A.astype(dt).ravel()).cuda()
            Bd = torch.from_numpy(np.ascontiguousarray(B.T).astype(dt)).cuda()  # column-major n x 2
            torch.cuda.synchronize()
            assert factor(wp, Ad.data_ptr(), n, st.cuda_stream) == 0
            assert solve(wp, Ad.data_ptr(), n, 2, Bd.data_ptr(), st.cuda_stream) == 0
            assert g.bem_lu_status(wp, st.cuda_stream) == 0
            X = Bd.cpu().numpy().T.astype(np.complex128)
            res.append(np.linalg.norm(A @ X - B) / (np.linalg.norm(A) * np.linalg.norm(X)))
    finally:
        g.bem_lu_free(wp)
    assert max(res) < (1e-13 if precision == "z" else 2e-6), res


@pytest.mark.parametrize("unload", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_context_solves_sizes_in_turn(unload, precision):
    """216, 600 and 216 quads again (n = 1728, 4800): the later small solve as the first."""
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    g.bemgpu_load.argtypes = [ctypes.c_void_p, ctypes.POINTER(api.Problem)]
    g.bemgpu_unload.argtypes = [ctypes.c_void_p]
    cases = [api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_lr_"), n=n, theta_deg=23.0,
                                                       phi_deg=41.0)) for n in (6, 10)]
    probs = [c.problem() for c in cases]
    ctx, got = ctypes.c_void_p(), []
    assert g.bemgpu_create(0, None, ctypes.byref(ctx)) == 0
    try:
        assert g.bemgpu_set_precision(ctx, precision) == 0
        for i in (0, 1, 0, 1):
            if unload:
                assert g.bemgpu_unload(ctx) == 0
            p, ne = probs[i], probs[i].Ne
            assert g.bemgpu_load(ctx, ctypes.byref(p)) == 0
            assert g.bemgpu_run(ctx) == 0, g.bemgpu_error(ctx)
            assert g.bemgpu_status(ctx) == 0
            out = [np.zeros((ne, 4), np.complex128) for _ in range(2)] + [np.zeros((ne, 4, 3), np.complex128) for _ in range(2)]
            assert g.bemgpu_get_solution(ctx, 0, *[api._p(x.view(np.float64)) for x in out]) == 0
            got.append(out)
    finally:
        g.bemgpu_destroy(ctx)
        for c, p in zip(cases, probs):
            c.free_problem(p)
            c.close()
    for a, b in zip(got[:2], got[2:]):
        for x, y in zip(a, b):
            assert np.max(np.abs(x - y)) <= (1e-13 if precision == 0 else 1e-12) * np.max(np.abs(x))
