"""The periodic domain's matrices from lattice images and an expansion of the
rest (the default of a context) against the lattice sums at every quadrature
point (the allocation-free entry point, which keeps them): G and H of bodies
over the forms that take the split: square, triangular and oblique lattices,
periods from where the body nearly fills its cell to more than three
wavelengths, spheres and spheroids as they stand, turned or off centre, meshes
of odd sizes (tile edges of the matrix product).

Tolerance (fixed before the first run): both sides carry the reference's sums to
1e-15 per term and agree with the converged integral of each entry to 1e-13
(the shorter rules' bound) or better; 1e-12 of the row's largest entry."""
import ctypes
import os
import sys
import tempfile

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_zz_no_alloc as static  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-12
SQ = ((1.0, 0.0), (0.0, 1.0))
TRI = ((1.0, 0.0), (0.5, 0.75 ** 0.5))
OBL = ((1.0, 0.0), (0.3, 0.9))
CASES = [  # n, radius, stretch, lattice, period, turned, centre
    (1, 0.2, 1.0, SQ, 0.8, False, (0, 0, 0)),
    (3, 0.3, 1.0, SQ, 0.8, True, (0, 0, 0.013)),
    (5, 0.29, 1.0, SQ, 0.7, True, (0.11, -0.07, 0.02)),
    (4, 0.31, 1.35, TRI, 0.72, False, (0, 0, 0)),
    (7, 0.25, 1.5, OBL, 1.0, True, (0, 0, 0.013)),
    (3, 0.35, 1.0, OBL, 3.3, True, (0, 0, 0.013)),
    (4, 0.2, 2.5, TRI, 1.1, True, (0, 0, 0)),
]


def _lattice(lat, a):
    return tuple(tuple(a * x for x in v) for v in lat)


@pytest.mark.parametrize("n,radius,stretch,lat,a,turned,centre", CASES)
@pytest.mark.parametrize("far_rule", [0, 1])
def test_split_matches_lattice_sums(n, radius, stretch, lat, a, turned, centre, far_rule):
    import torch
    from bem3_aw_qd2_b200 import api, meshgen
    api.libs()[0].aqd2_set_verbose(0)
    d = tempfile.mkdtemp(prefix="bem_split_")
    kw = dict(rot=((1.0, 2.0, 3.0), 37.0)) if turned else {}
    case = api.Case.from_files(*meshgen.write_inputs(d, n=n, semi_axes=(radius, radius, radius * stretch),
                                                     lattice=_lattice(lat, a), center=centre, theta_deg=23.0,
                                                     phi_deg=41.0, **kw))
    case.solve()
    case.set_far_rule(far_rule)
    case.run_device()
    assert case.status() == 0
    path = os.path.join(d, "c.dat")
    case.dat_write(path)
    t = static.parse_dat(path)
    dev = torch.device("cuda:0")
    for k in ("cr", "cw", "ren", "plane"):
        t[k + "_d"] = torch.tensor(t[k], device=dev)
    o = static._static_matrices(static._entry(), t, 0, torch.cuda.Stream(device=dev), dev)
    N = 24 * n * n
    for k in ("G", "H"):
        got, ref = case.matrix(0, k, N), o[k].cpu().numpy()
        err = np.max(np.abs(got - ref) / np.max(np.abs(ref), axis=1, keepdims=True))
        assert err < TOL, (k, err)
    case.close()


def test_selected_batch_instance_assembles_alone():
    """bemgpu_assemble while a batch is loaded assembles the selected instance:
    its own Bloch phases, not instance 0's."""
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    cases = [api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_sel_"), n=3, theta_deg=th, phi_deg=ph))
             for th, ph in ((20.0, 30.0), (35.0, 10.0), (50.0, 200.0))]
    probs = [c.problem() for c in cases]
    g.bemgpu_load.argtypes = [ctypes.c_void_p, ctypes.POINTER(api.Problem)]
    g.bemgpu_batch_load.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.POINTER(api.Problem))]
    g.bemgpu_batch_select.argtypes = [ctypes.c_void_p, ctypes.c_int]
    ctx = ctypes.c_void_p()
    assert g.bemgpu_create(0, None, ctypes.byref(ctx)) == 0
    N = 216

    def matrices():
        out = []
        for w in (0, 1):
            m = np.zeros((N, N), np.complex128)
            assert g.bemgpu_get_matrix(ctx, 0, w, api._p(m.view(np.float64))) == 0
            out.append(m)
        return out
    try:
        assert g.bemgpu_load(ctx, ctypes.byref(probs[2])) == 0 and g.bemgpu_assemble(ctx) == 0
        ref = matrices()
        arr = (ctypes.POINTER(api.Problem) * 3)(*[ctypes.pointer(p) for p in probs])
        assert g.bemgpu_batch_load(ctx, 3, arr) == 0
        assert g.bemgpu_batch_select(ctx, 2) == 0 and g.bemgpu_assemble(ctx) == 0
        for x, y in zip(matrices(), ref):
            assert np.max(np.abs(x - y)) <= 1e-13 * np.max(np.abs(y))
    finally:
        g.bemgpu_destroy(ctx)
        for c, p in zip(cases, probs):
            c.free_problem(p)
            c.close()
