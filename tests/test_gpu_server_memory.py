"""What the server counts for a problem: the buffers of the periodic domain's split grow
with its degree, so that of two bodies of as many elements the one that nearly fills its
cell counts more, by what the larger degree's matrix alone takes; and the count covers
what the device gives away for it.

Degrees of these bodies on 24 elements: 16 (K = 289) and 26 (K = 729): the matrices T of K
x 2 K doubles, K rounded up to 16, differ by 7.19 MB."""
import tempfile

import pytest

pytestmark = pytest.mark.gpu


def test_count_holds_the_split():
    import torch
    from bem3_aw_qd2_b200 import api, meshgen
    api.libs()[0].aqd2_set_verbose(0)
    bodies = [dict(semi_axes=(0.16,) * 3, lattice=((1.6, 0.0), (0.0, 1.6))),
              dict(semi_axes=(0.28, 0.28, 0.5), lattice=((0.7, 0.0), (0.0, 0.7)))]
    cases = [api.Case.from_files(*meshgen.write_inputs(tempfile.mkdtemp(prefix="bem_sm_"), n=2, theta_deg=23.0, phi_deg=41.0,
                                                       rot=((1.0, 2.0, 3.0), 37.0), **b)) for b in bodies]
    probs = [c.problem() for c in cases]
    counted, taken = [], []
    try:
        for i, p in enumerate(probs):
            srv = api.Server(slots=1, hbm_budget=8 << 30)
            free0 = torch.cuda.mem_get_info(0)[0]
            srv.submit(p, 77 + i, i)
            done = []
            while not done:
                done = srv.poll()
            assert done[0].status == 0, done[0].error
            counted.append(srv.stats()["bytes_resident"])
            taken.append(free0 - torch.cuda.mem_get_info(0)[0])
            srv.close()
    finally:
        for c, p in zip(cases, probs):
            c.free_problem(p)
            c.close()
    assert counted[1] - counted[0] > 7.1e6, counted
    assert all(t <= c for t, c in zip(taken, counted)), (taken, counted)
