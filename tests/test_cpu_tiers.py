"""Error model of the shorter rules away from the reference's 12 x 12 (no GPU),
for the two threshold tables beside the periodic pairs' own (bem_tiers.cuh):

  tier_free    free space with the tangential derivatives of G and H, and the
               geometric sums: 10 points from 4 R, 9 from 5, 8 from 7, 7 from 9
               (k R <= 0.5), 6 from 16 (k R <= 0.25): 1e-14 of the largest entry of
               each matrix (G, H, dG, dH), the rounding of a 144-point sum;
  tier_image   G and H of one image of the periodic domain: 10 from 3, 9 from 3.5,
               8 from 5, 7 from 7, 6 from 12 (k R <= 0.5): 2e-13 of its largest.

Bilinear quads inside the shape guard (twist at most a tenth of the shorter
half-side, sides within 3x) and triangles with angles of 25 degrees and more,
seeded directions, against a 28-point rule."""
import numpy as np
import pytest

SQ3 = np.sqrt(3.0)
FREE = [(10, 4, 1.0), (9, 5, 1.0), (8, 7, 1.0), (7, 9, 0.5), (6, 16, 0.25)]
IMAGE = [(10, 3, 1.0), (9, 3.5, 1.0), (8, 5, 1.0), (7, 7, 0.5), (6, 12, 0.5)]


def kernels(k, R, W, v1, v2):
    a = np.linalg.norm(R, axis=-1)
    e, cb = np.exp(1j * k * a), 1j * k * a - 1
    aW, rW = np.linalg.norm(W, axis=-1), (R * W).sum(-1) / a
    out = [e / a * aW, cb * e * rW / a ** 2]
    for v in (v1, v2):
        rv, Wv = (R @ v) / a, W @ v
        out += [cb * e / a ** 2 * rv * aW, e * ((k * k * a * a + 3 * cb) * rv * rW - cb * Wv) / a ** 3]
    return out


def quad(n, k, t, tw, asp, v):
    x, w = np.polynomial.legendre.leggauss(n)
    X, Y = np.meshgrid(x, x, indexing="ij")
    o = 0 * X
    r = np.stack([X, asp * Y, tw * X * Y], -1)
    W = np.cross(np.stack([o + 1, o, tw * Y], -1), np.stack([o, o + asp, tw * X], -1))
    N = [0.25 * (1 + a * X * SQ3) * (1 + b * Y * SQ3) for a, b in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
    return np.array([[np.sum(np.outer(w, w) * f * Na) for Na in N] for f in kernels(k, r - t, W, *v)])


def tri(n, k, t, C, v):
    x, w = np.polynomial.legendre.leggauss(n)
    u = 0.5 * (x + 1)
    U, V = np.meshgrid(u, u, indexing="ij")
    z, e = 1 - 1.5 * U, 0.5 * SQ3 * U * (1 - 2 * V)
    r = z[..., None] * C[0] + e[..., None] * C[1]
    W = np.cross(C[0], C[1]) + 0 * r
    N = [1 / 3 * (1 - 2.5 * (z + SQ3 * e)), 1 / 3 * (1 + 5 * z), 1 / 3 * (1 - 2.5 * (z - SQ3 * e))]
    return np.array([[np.sum(np.outer(w, w) * U * f * Na) for Na in N] for f in kernels(k, r - t, W, *v)])


def worst(n, d, kR, kind, rows, seed):
    rng = np.random.default_rng(seed)
    bad = 0.0
    for it in range(40):
        v1 = rng.normal(size=3)
        v1 /= np.linalg.norm(v1)
        v2 = np.cross(v1, rng.normal(size=3))
        v2 /= np.linalg.norm(v2)
        u = rng.normal(size=3)
        if it % 3 == 0:
            u[2] *= 0.1
        u /= np.linalg.norm(u)
        if kind == "quad":
            asp = rng.choice([1.0, 1 / 3, 0.6])
            tw = rng.uniform(-0.1, 0.1) * asp
            R = np.sqrt(1 + asp ** 2 + tw ** 2 + 2 * abs(tw) * 0)
            f = lambda m: quad(m, kR / R, u * d * R, tw, asp, (v1, v2))  # noqa: E731
            area = 4 * asp
        else:
            while True:
                p = rng.normal(size=(3, 3))
                p -= p.mean(0)
                a = [np.linalg.norm(p[i] - p[j]) for i, j in ((0, 1), (1, 2), (2, 0))]
                ang = [np.degrees(np.arccos((a[i] ** 2 + a[(i + 2) % 3] ** 2 - a[(i + 1) % 3] ** 2) /
                                            (2 * a[i] * a[(i + 2) % 3]))) for i in range(3)]
                if min(ang) >= 25:
                    break
            R = 1.0
            p /= np.linalg.norm(p, axis=1).max()
            C = (p[0], (p[1] - p[2]) / SQ3)
            f = lambda m: tri(m, kR, u * d, C, (v1, v2))  # noqa: E731
            area = np.linalg.norm(np.cross(*C))
        got, ref = f(n), f(28)
        for idx in rows:
            # an entry that vanishes by geometry (H in the plane) counts against a tenth of the kernel's size
            size = 0.1 * area / 4 * (d * R) ** -{0: 1, 1: 2, 2: 2, 3: 3}[idx[0]]
            bad = max(bad, np.abs(got[idx] - ref[idx]).max() / max(np.abs(ref[idx]).max(), size))
    return bad


@pytest.mark.parametrize("kind", ["quad", "tri"])
@pytest.mark.parametrize("n,d,kR", FREE)
def test_free_space_rules(n, d, kR, kind):
    for k in (0.2 * kR, kR):
        assert worst(n, d, k, kind, ([0], [1], [2, 4], [3, 5]), seed=n) < 1e-14


@pytest.mark.parametrize("n,d,kR", IMAGE)
def test_image_rules(n, d, kR):
    for k in (0.2 * kR, kR):
        assert worst(n, d, k, "quad", ([0], [1]), seed=10 + n) < 2e-13
