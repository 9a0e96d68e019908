"""Field sums of many points above the body, out to 60 wavelengths: there the lattice
sums are few plane waves, no split of the lattice reaches the points, and finding that
out must cost little beside the sums (a list of every lattice point out to the points
took 10 to 150 ms of host time a call).  Values against the same points one call at a
time; the call's time as a whole.

Tolerance (fixed before the first run): the same sums, the nearer heights' spectral
orders from a table instead of directly: 1e-12 of the largest value.  Time: the sums of
2000 points of 216 quads on the 9-point rule take 1 to 4 ms at these heights; the
median of five calls stays below 6 ms."""
import ctypes
import tempfile
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [1.5, 4.0, 12.0, 60.0])
@pytest.mark.parametrize("kind", [1, 0x101])
def test_far_points(height, kind):
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    case = api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_ff_"), n=6, theta_deg=23.0, phi_deg=41.0,
                                                     rot=((1.0, 2.0, 3.0), 37.0)))
    case.solve()
    g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
    rng = np.random.default_rng(5)
    n = 2000
    r = rng.uniform(-0.4, 0.4, (n, 3))
    r[:, 2] = np.where(rng.random(n) < 0.5, -1.0, 1.0) * (height + 0.05 * rng.random(n))
    out, t = np.zeros((n, 18)), []
    for _ in range(5):
        t0 = time.perf_counter()
        assert g.bemgpu_field(case.ctx, 0, kind, n, api._p(r), api._p(out)) == 0
        t.append(time.perf_counter() - t0)
    some = range(0, n, 97)
    one = np.zeros((len(some), 18))
    for i, p in enumerate(some):
        x, y = np.ascontiguousarray(r[p]), np.zeros(18)
        assert g.bemgpu_field(case.ctx, 0, kind, 1, api._p(x), api._p(y)) == 0
        one[i] = y
    case.close()
    for c in (slice(0, 2), slice(2, 8), slice(12, 18)):
        assert np.max(np.abs(out[some][:, c] - one[:, c])) <= 1e-12 * np.max(np.abs(one[:, c]))
    assert sorted(t)[2] < 6e-3, t
