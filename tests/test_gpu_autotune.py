"""The Ewald autotuner times the lattice-sum kernels where the assembly runs them, and
times nothing where images and expansion stand in their place: then it sets the rule's
scale, 0.98 sqrt(3) / (k eta0) clamped to [0.5, 1.3] (the square lattice's eta0 is its
period / sqrt(4 pi)).  Either way the tuned problem solves to the same force.

Tolerance: both lattice sums converge to 1e-15 for any scale; 1e-9 of the force, as the
reference systems hold it."""
import math
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axes,period,split", [((0.3, 0.3, 0.3), 0.8, True), ((0.3, 0.3, 1.2), 0.7, False)])
def test_times_what_runs(axes, period, split):
    from bem3_aw_qd2_b200 import api, meshgen
    h, g = api.libs()
    h.aqd2_set_verbose(0)
    case = api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_at_"), n=2, semi_axes=axes, theta_deg=23.0,
                                                     phi_deg=41.0, lattice=((period, 0.0), (0.0, period))))
    case.solve()
    F0, _ = case.force()
    n0 = g.bemgpu_kernel_launches()
    scale = case.autotune()
    launched = g.bemgpu_kernel_launches() - n0
    rule = min(max(0.98 * math.sqrt(3.0) / (2.0 * math.pi * period / math.sqrt(4.0 * math.pi)), 0.5), 1.3)
    if split:
        assert launched <= 2 and abs(scale - rule) < 1e-12 * rule, (launched, scale, rule)  # the tables of that scale
    else:
        assert launched > 20, launched  # four candidates, each timed twice
        assert any(abs(scale - x) < 1e-12 * x for x in (rule, 0.9 * rule, 0.8 * rule, 1.0 if rule < 1.0 else 1.1 * rule))
    case.run_device()
    F1, _ = case.force()
    case.close()
    assert np.max(np.abs(F1 - F0)) <= 1e-9 * np.max(np.abs(F0))
