"""Which field calls build a spectral order table that reaches out to their points, and
their values: many points over a flat body on a sparse lattice (the mesh's own table
holds few of the heights that matter) build one; points high above it, where plane
waves alone do, points of a lattice whose Ewald parameter is capped next to the body, and
a single point of a small mesh do not.  Values against the same points one call at a
time, both sums (with and without second derivatives).

Tolerance (fixed before the first run): the tables carry each order to 1e-16 of its
interval's scale, some 100 terms a sum: 1e-12 of the largest value."""
import ctypes
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("period,axes,height,table", [
    (1.6, (0.3, 0.3, 0.05), 0.1, 1), (1.6, (0.3, 0.3, 0.05), 0.5, 1), (1.6, (0.3, 0.3, 0.05), 3.0, 0),
    (3.3, (0.35, 0.35, 0.35), 0.5, 0), (0.8, (0.3, 0.3, 0.3), 0.32, 0)])
@pytest.mark.parametrize("kind", [1, 0x101])
def test_table_where_it_serves(period, axes, height, table, kind):
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    case = api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_fr_"), n=2, semi_axes=axes, theta_deg=23.0,
                                                     phi_deg=41.0, lattice=((period, 0.0), (0.0, period))))
    case.solve()
    g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
    rng = np.random.default_rng(5)
    n = 1200  # three waves of blocks, below the calls that images and expansion are planned for
    r = rng.uniform(-0.4, 0.4, (n, 3))
    r[:, 2] = np.where(rng.random(n) < 0.5, -1.0, 1.0) * (height + 0.05 * rng.random(n))
    out = np.zeros((n, 18))
    n0 = g.bemgpu_kernel_launches()
    assert g.bemgpu_field(case.ctx, 0, kind, n, api._p(r), api._p(out)) == 0
    assert g.bemgpu_kernel_launches() - n0 == table
    some = range(0, n, 97)
    one = np.zeros((len(some), 18))
    n0 = g.bemgpu_kernel_launches()
    for i, p in enumerate(some):
        x, y = np.ascontiguousarray(r[p]), np.zeros(18)
        assert g.bemgpu_field(case.ctx, 0, kind, 1, api._p(x), api._p(y)) == 0
        one[i] = y
    assert g.bemgpu_kernel_launches() == n0
    case.close()
    for c in (slice(0, 2), slice(2, 8), slice(8, 9), slice(9, 12), slice(12, 18)):
        assert np.max(np.abs(out[some][:, c] - one[:, c])) <= 1e-12 * np.max(np.abs(one[:, c]))
