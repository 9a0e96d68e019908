"""Truncation of the expansion that stands for the lattice images left out of
the closed forms (no GPU): an image at distance c from the body's centre, seen
from collocation points and source points within R0 of it, is
  e^{ikd}/d = ik sum_l (2l + 1) j_l(k|y|) h_l(k|D|) P_l(cos),   D = image - x,
cut at the degree the host picks: the smallest whose later terms stay below
1e-15 of 1 / (2 R0), six images counted (bem_smooth.cu, degree_for).  Over the
ranges of c / R0 and k R0 that take the split, the cut sum agrees with the
closed form, value and gradient along y, to 1e-14 of 1 / (2 R0)."""
import math

import numpy as np
import pytest


def _j(n, z):
    top = n + 20 + int(4 * z)  # far enough up that the starting series does not cancel
    g = np.zeros(top + 2)
    for l in (top, top + 1):
        t = s = 1.0
        for m in range(1, 200):
            t *= -0.5 * z * z / (m * (2 * l + 2 * m + 1))
            s += t
        g[l] = s
    for l in range(top, 0, -1):
        g[l - 1] = g[l] - z * z / ((2 * l + 1) * (2 * l + 3)) * g[l + 1]
    f, j = 1.0, np.zeros(n + 1)
    for l in range(n + 1):
        j[l] = f * g[l]
        f *= z / (2 * l + 3)
    return j


def _h(n, z):
    y = np.zeros(n + 2)
    y[0], y[1] = -math.cos(z) / z, -math.cos(z) / z ** 2 - math.sin(z) / z
    for l in range(1, n + 1):
        y[l + 1] = (2 * l + 1) / z * y[l] - y[l - 1]
    return _j(n, z) + 1j * y[:n + 1]


def _degree(k, a, b, scale, tol=1e-15, lim=60):
    j, h = _j(lim + 4, k * a), np.abs(_h(lim + 4, k * b))
    for l in range(lim, -1, -1):
        if k * (2 * l + 3) * abs(j[l + 1]) * h[l + 1] * scale > tol:
            return l + 1
    return 0


@pytest.mark.parametrize("kR0", [0.3, 1.9, 2.8, 5.0])
@pytest.mark.parametrize("ratio", [2.2, 2.7, 4.0, 9.0])
def test_truncated_image_matches_closed_form(kR0, ratio):
    k = 2 * np.pi
    R0 = kR0 / k
    c = ratio * R0
    L = _degree(k, R0, c - R0, 12.0 * R0)
    rng = np.random.default_rng(1)
    worst = 0.0
    for _ in range(200):
        u = rng.normal(size=(2, 3))
        u /= np.linalg.norm(u, axis=1)[:, None]
        y = u[0] * R0 * rng.uniform(0.3, 1.0)
        D = np.array([c, 0, 0]) - u[1] * R0 * rng.uniform(0.0, 1.0)
        ry, rD = np.linalg.norm(y), np.linalg.norm(D)
        x = y @ D / (ry * rD)
        j, h = _j(L, k * ry), _h(L, k * rD)
        P = np.polynomial.legendre.legvander(np.array([x]), L)[0]
        got = 1j * k * np.sum((2 * np.arange(L + 1) + 1) * j * h * P)
        d = np.linalg.norm(D - y)
        worst = max(worst, abs(got - np.exp(1j * k * d) / d) * 2 * R0)
    assert worst < 1e-14, worst
