"""The LU's panels at the edges of their tournament (slices of 256 rows, up to
eight winners' lists per next level: one level to 256 rows, two to 2048, three
beyond) and of their sub-blocks of eight columns (last panels of 1 to 31
columns), rows out of order so that every level hands pivots on, rows that
repeat in size (ties of the pivot search), and a matrix that is singular only
in its last columns.  Tolerance: 1e-13 for the residual relative to ||A|| ||X||,
as the other sizes of bemgpu_zgesv are held to (test_gpu_lu.py)."""
import numpy as np
import pytest

from test_gpu_lu import random_system, zgesv

pytestmark = pytest.mark.gpu


def _residual(A, X, B):
    return np.linalg.norm(A @ X - B) / (np.linalg.norm(A) * np.linalg.norm(X))


@pytest.mark.parametrize("n", [8, 9, 40, 256, 263, 512, 520, 2047, 2048, 2049, 2337])
def test_tournament_edges(n):
    A, B = random_system(n, 1, seed=31 + n, permuted=True)
    rc, X = zgesv(A, B)
    assert rc == 0
    assert _residual(A, X, B) < 1e-13


@pytest.mark.parametrize("n", [48, 300])
def test_ties_of_the_pivot_search(n):
    # entries of one modulus sum |re| + |im|: every key of the first column is equal
    rng = np.random.default_rng(n)
    A = rng.choice([1.0, -1.0], (n, n)) + 1j * rng.choice([1.0, -1.0], (n, n))
    B = rng.standard_normal((n, 2)) + 0j
    rc, X = zgesv(A, B)
    assert rc == 0
    assert _residual(A, X, B) < 1e-13


@pytest.mark.parametrize("n", [33, 300])
def test_zero_row_is_reported(n):
    A, B = random_system(n, 1, seed=3)
    A[n // 2] = 0.0  # its pivot is the last one, exactly zero
    assert zgesv(A, B)[0] == -3
