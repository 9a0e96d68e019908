"""The triangular solves (k_lu_trsv through bemgpu_zgesv) at the edges of their
32-row blocks, for each number of right-hand sides: one block, two, a last block
of one row, of 31; against numpy's LAPACK solve.  A right-hand side of all-ones
NaN words, the pattern that the solves reserve for values not yet written, gives
NaN and nothing else.

Tolerance (fixed before the first run): the matrices' condition numbers stay
below 1e3 (diagonal 1.5 over entries of 1 / sqrt(n)): 1e-11 of the solution."""
import numpy as np
import pytest

from test_gpu_lu import random_system, zgesv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 97, 417])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4])
def test_block_edges(n, nrhs):
    A, B = random_system(n, nrhs, seed=31 * n + nrhs, permuted=True)
    rc, X = zgesv(A, B)
    assert rc == 0
    ref = np.linalg.solve(A, B)
    assert np.linalg.norm(X - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [5, 100])
def test_reserved_pattern_in_the_right_hand_side(n):
    A, B = random_system(n, 2, seed=n)
    B = np.asfortranarray(B)
    B[:, 1].view(np.uint64)[:] = 0xFFFFFFFFFFFFFFFF
    rc, X = zgesv(A, B)
    assert rc == 0
    assert np.all(np.isnan(X[:, 1]))
    ref = np.linalg.solve(A, B[:, 0])
    assert np.linalg.norm(X[:, 0] - ref) <= 1e-11 * np.linalg.norm(ref)
