"""Field sums of many points, whose spectral order table reaches out to the
points, against the same points one call at a time (a single point does not pay
for a table: its terms beyond the context's own table are evaluated directly).
Heights from beside the body to where the plane-wave sum takes over, above and
below; both sums (with and without second derivatives).

Tolerance (fixed before the first run): the tables carry each order to 1e-16 of
its interval's scale, some 100 terms a sum: 1e-12 of the largest value."""
import ctypes
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("potential", [0, 0x100])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("height", [0.0, 0.31, 0.7, 1.6, 4.0])
def test_table_of_many_points_matches_single_points(potential, kind, height):
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    case = api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_ft_"), n=2, theta_deg=23.0, phi_deg=41.0))
    case.solve()
    g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
    rng = np.random.default_rng(5)
    n = 2000
    r = rng.uniform(-0.4, 0.4, (n, 3))
    rho = np.hypot(r[:, 0], r[:, 1])
    r[:, :2] *= (np.maximum(rho, 0.34) / rho)[:, None]  # outside the body
    r[:, 2] = np.where(rng.random(n) < 0.5, -1.0, 1.0) * (height + 0.05 * rng.random(n))
    out = np.zeros((n, 18))
    assert g.bemgpu_field(case.ctx, 0, kind | potential, n, api._p(r), api._p(out)) == 0
    some = range(0, n, 97)
    one = np.zeros((len(some), 18))
    for i, p in enumerate(some):
        x, y = np.ascontiguousarray(r[p]), np.zeros(18)
        assert g.bemgpu_field(case.ctx, 0, kind | potential, 1, api._p(x), api._p(y)) == 0
        one[i] = y
    case.close()
    for c in (slice(0, 2), slice(2, 8), slice(8, 9), slice(9, 12), slice(12, 18)):
        assert np.max(np.abs(out[some][:, c] - one[:, c])) <= 1e-12 * np.max(np.abs(one[:, c]))
