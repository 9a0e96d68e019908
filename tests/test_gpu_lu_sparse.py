"""Matrices with many zeros through the dense solve: a panel's rows are chosen in slices,
and a slice whose rows are zero in the panel's first columns must still hand on the
rows that later columns need.  Permutation matrices whose panels have their pivots in
different slices, permuted block-diagonal and banded matrices, against numpy's LAPACK.

Tolerance: a permutation's solution is exact; else the residual relative to ||A|| ||X||
as test_gpu_lu.py holds it, 1e-13."""
import numpy as np
import pytest

from test_gpu_lu import zgesv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [257, 600, 2100, 2500])
@pytest.mark.parametrize("order", ["halves", "reverse", "shift"])
def test_permutation(n, order):
    # halves: the first 16 columns of a panel pivot in the first slice, the others near the end
    j = np.arange(n)
    rows = {"reverse": j[::-1], "shift": (j + 7 * n // 16) % n,
            "halves": np.concatenate([j[(j // 16) % 2 == 0], j[(j // 16) % 2 == 1]]).argsort()}[order]
    A = np.zeros((n, n), np.complex128)
    A[rows, j] = np.exp(1j * j)
    B = (np.arange(1, 2 * n + 1) * (0.5 - 0.25j)).reshape(2, n).T
    rc, X = zgesv(A, B)
    assert rc == 0
    assert np.max(np.abs(X - np.exp(-1j * j)[:, None] * B[rows])) <= 1e-12 * np.max(np.abs(B))


@pytest.mark.parametrize("n,width", [(600, 16), (600, 40), (2500, 24)])
@pytest.mark.parametrize("kind", ["block", "band"])
def test_zeros_between_blocks(n, width, kind):
    rng = np.random.default_rng(n + width)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    i, j = np.indices((n, n))
    A[(i // width != j // width) if kind == "block" else (np.abs(i - j) > width)] = 0.0
    A += np.eye(n) * 8.0 * np.sqrt(width)
    A = A[rng.permutation(n)]
    B = rng.standard_normal((n, 2)) + 0j
    rc, X = zgesv(A, B)
    assert rc == 0
    assert np.linalg.norm(A @ X - B) / (np.linalg.norm(A) * np.linalg.norm(X)) < 1e-13
