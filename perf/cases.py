"""Performance cases: the calls that a user of this library makes, over the
sizes, meshes, lattices and precisions that it is used at.

A case is a dict of plain values.  `kind` names the call:

  solve     solve_bieq_aqd2 + force_FN_aqd2 (Case.solve, Case.force): one
            boundary-value problem from its element tables to P, dP, pv, dpv of
            both domains and the radiation force; `precision` 0 is the FP64
            drop-in, 2 the mixed form (TF32 tensor-core updates, FP64 refinement).
            Every pass assembles and factors every domain (interior reuse off),
            on a resident device context, as a program that solves one body
            after another does.
  sweep     a batch of incidence directions on one body and frequency
            (bemgpu_batch_load / _assemble / _select / solve / force)
  incident  a new incident field on kept factors (bemgpu_set_incident,
            bemgpu_solve_rhs, force): a repeated request of the server
  force9    the 9-point (triangles: 7-point) radiation force of a solved body
  field     pressure and velocity sums on a grid of points around a solved body
  point     pressure and velocity at one point (pv_t_aqd2)
  greens    the quasi-periodic Green's function and its gradient at points
  dense     the dense complex solve (bemgpu_zgesv) on host arrays

Bodies are the cube-spheres, spheroids (bilinear quads, 6 n^2 elements) and
icospheres (triangles, 20 4^level) of meshgen, radius 0.2 to 0.35 wavelengths,
as they stand or turned about a generic axis; lattices are square, triangular
or oblique with periods of 0.7 to 1.1 wavelengths, up to 3.3 for the sparse ones
of the reference's verification runs.  The seed draws the direction of incidence
and the body's medium.
"""
import ctypes
import math
import random
import shutil
import tempfile

import numpy as np

from bem3_aw_qd2_b200 import api, meshgen

KINDS = ("solve", "sweep", "incident", "force9", "field", "point", "greens", "dense")


def listed():
    def body(name, kind, n, **more):
        c = dict(name=name, kind=kind, mesh="quad", n=n, radius=0.3, stretch=1.0, lattice="square", period=0.8,
                 turned=False, precision=0)
        c.update(more)
        return c

    return [
        # the smallest solve: latency of the whole path (smoke and fixture size)
        body("solve24", "solve", 2),
        # the benchmark's own workload
        body("solve216", "solve", 6),
        # the size of the reference's shipped examples (600 quads, period of one
        # wavelength, triangular lattice), body in a general position
        body("solve600", "solve", 10, radius=0.333, lattice="triangular", period=1.0, turned=True),
        # the largest FP64 solve: the body of the direction sweeps
        body("solve1536", "solve", 16),
        # triangle meshes
        body("solve_tri320", "solve", 2, mesh="tri", lattice="triangular"),
        # mixed precision at the size where it is used, a spheroid on an oblique lattice
        body("mixed1014", "solve", 13, radius=0.25, stretch=1.5, lattice="oblique", period=1.0, turned=True,
             precision=2),
        # eight directions on the 216-quad sphere
        body("sweep216", "sweep", 6, count=8),
        # a repeated request on a large resident body
        body("incident726", "incident", 11, turned=True),
        # post-processing of a solved body
        body("force9_150", "force9", 5, turned=True),
        body("field216", "field", 6, count=1500),
        # the point evaluator behind every sum
        dict(name="greens20k", kind="greens", lattice="oblique", period=0.9, count=20000),
        # the dense solver on its own, three right-hand sides
        dict(name="dense1999", kind="dense", n=1999, count=3),
    ]


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "solve", "mixed", "sweep", "incident", "force9", "field", "point",
                       "greens", "dense"))
    lattice = rng.choice(("square", "triangular", "oblique"))
    period = round(rng.uniform(0.7, 1.1), 3) if rng.random() < 0.8 else round(rng.uniform(1.1, 3.3), 3)

    def size(lo, hi):  # integers spread over their logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "greens":
        return dict(kind=kind, lattice=lattice, period=period, count=size(100, 40000))
    if kind == "dense":
        return dict(kind=kind, n=size(50, 3000), count=rng.choice((1, 2, 3, 4)))
    mixed = kind == "mixed"
    c = dict(kind="solve" if mixed else kind, lattice=lattice, period=period, turned=rng.random() < 0.5,
             precision=2 if mixed else 0)
    # the 9-point rule on a mesh with mirrored elements meets the lattice plane
    # of its own targets, where the reference's sums stop on rounding noise:
    # its bodies are turned
    tri = kind not in ("sweep", "force9") and rng.random() < 0.25
    if kind == "force9":
        c["turned"] = True
    c["mesh"] = "tri" if tri else "quad"
    if tri:
        c["n"] = rng.choice((1, 2, 3) if kind == "solve" else (1, 2))
        c["turned"] = False
    elif kind == "solve":
        c["n"] = size(2, 15)
    elif mixed:
        c["n"] = size(6, 15)
    elif kind == "incident":
        c["n"] = size(4, 13)
    else:
        c["n"] = size(2, 8)
    c["stretch"] = rng.choice((1.0, 1.0, 1.35, 1.5))
    # the body fits its cell with a gap
    c["radius"] = round(min(rng.uniform(0.2, 0.35), 0.42 * period / (c["stretch"] if c["turned"] else 1.0)), 3)
    if kind == "sweep":
        c["count"] = rng.choice((2, 3, 5, 8))
    elif kind == "field":
        c["count"] = size(20, 2000)
    return c


# ---------------------------------------------------------------- inputs
def _lattice(case):
    a = case["period"]
    return {"square": ((a, 0.0), (0.0, a)), "triangular": ((a, 0.0), (0.5 * a, 0.5 * math.sqrt(3.0) * a)),
            "oblique": ((a, 0.0), (0.3 * a, 0.9 * a))}[case["lattice"]]


def _reciprocal(lat):
    (ax, ay), (bx, by) = lat
    f = 2.0 * math.pi / (ax * by - bx * ay)
    return (f * by, -f * bx), (-f * ay, f * ax)


def _direction(lat, rng):
    """Angles of incidence (degrees) at least 2 % away from a Rayleigh anomaly (unit wavelength)."""
    k = 2.0 * math.pi
    g1, g2 = _reciprocal(lat)
    while True:
        th, ph = rng.uniform(5.0, 60.0), rng.uniform(0.0, 360.0)
        kx = k * math.sin(math.radians(th)) * math.cos(math.radians(ph))
        ky = k * math.sin(math.radians(th)) * math.sin(math.radians(ph))
        if abs(kx) > 1e-3 and abs(ky) > 1e-3 and all(
                abs(math.hypot(kx + i * g1[0] + j * g2[0], ky + i * g1[1] + j * g2[1]) - k) >= 0.02 * k
                for i in range(-8, 9) for j in range(-8, 9)):
            return th, ph, kx, ky


def _elements(case):
    return 20 * 4 ** case["n"] if case["mesh"] == "tri" else 6 * case["n"] ** 2


class _Body:
    """An initialised problem, and after solve() its resident device context."""

    def __init__(self, case, theta, phi, rho, c, amp=(1.0, 0.0)):
        api.libs()[0].aqd2_set_verbose(0)
        r = case["radius"]
        kw = dict(ico=case["n"]) if case["mesh"] == "tri" else dict(n=case["n"])
        if case["turned"]:
            kw["rot"] = ((1.0, 2.0, 3.0), 37.0)
            kw["center"] = (0.0, 0.0, 0.013)
        d = tempfile.mkdtemp(prefix="perf_case_")
        files = meshgen.write_inputs(d, semi_axes=(r, r, r * case["stretch"]), lattice=_lattice(case), theta_deg=theta,
                                     phi_deg=phi, rho_in=rho * meshgen.RHO0, c_in=c * meshgen.C0, amp=amp, **kw)
        self.case = api.Case.from_files(*files)
        shutil.rmtree(d)
        self.ne = _elements(case)
        self.pr = None

    def problem(self):
        if self.pr is None:
            self.pr = self.case.problem()
        return self.pr

    def __del__(self):
        if self.pr is not None:
            self.case.free_problem(self.pr)
        self.case.close()


def _solution(ctx, ne):
    """P, dP, pv, dpv of both domains on the host."""
    g = api.libs()[1]
    out = []
    for d in (0, 1):
        a = [np.zeros((ne, 4), np.complex128), np.zeros((ne, 4), np.complex128), np.zeros((ne, 4, 3), np.complex128),
             np.zeros((ne, 4, 3), np.complex128)]
        _ok(ctx, g.bemgpu_get_solution(ctx, d, *[api._p(x.view(np.float64)) for x in a]))
        out += a
    return out


def _ok(ctx, rc):
    if rc != 0:
        raise RuntimeError(api.libs()[1].bemgpu_error(ctx).decode())


def _force(ctx, kind=0, rc=(0.0, 0.0, 0.0)):
    """Force and torque about rc, one array (the torque of a sphere is round-off beside its force)."""
    g = api.libs()[1]
    o, rc = np.zeros(6), np.array(rc, dtype=np.float64)
    _ok(ctx, g.bemgpu_force(ctx, kind, api._p(rc), api._p(o), api._p(o[3:])))
    return o


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "dense":
        r = np.random.default_rng(seed)
        n, m = case["n"], case["count"]
        # rows of the size of a boundary-integral system's: a unit-scale diagonal over a decaying rest
        a = (r.standard_normal((n, n)) + 1j * r.standard_normal((n, n))) / math.sqrt(n)
        a[np.arange(n), r.permutation(n)] += 1.0 + 2.0 * r.random(n)
        b = r.standard_normal((m, n)) + 1j * r.standard_normal((m, n))
        f = api.libs()[1].bemgpu_zgesv
        f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, api._d, api._d]
        return dict(kind=kind, a=a, b=b, n=n, m=m)
    lat = _lattice(case)
    th, ph, kx, ky = _direction(lat, rng)
    if kind == "greens":
        k = 2.0 * math.pi
        kz = math.sqrt(k * k - kx * kx - ky * ky)
        r = np.random.default_rng(seed)
        n = case["count"]
        # differences of points of a body: across the cell and beyond, either side of the plane
        p = r.uniform(-0.7, 0.7, (n, 3)) * case["period"]
        p[:, 2] = r.uniform(0.04, 0.7, n) * np.where(r.random(n) < 0.5, -1.0, 1.0)
        return dict(kind=kind, qp=np.array([k, kx, ky, kz, *lat[0], *lat[1]]), r=p)
    rho, c = rng.uniform(1.1, 1.3), rng.uniform(1.2, 1.7)
    g = api.libs()[1]
    b = _Body(case, th, ph, rho, c)
    s = dict(kind=kind, body=b)
    if kind == "sweep":
        s["bodies"] = [b] + [_Body(case, *_direction(lat, rng)[:2], rho, c) for _ in range(case["count"] - 1)]
        P = ctypes.POINTER(api.Problem)
        s["probs"] = (P * case["count"])(*[ctypes.pointer(x.problem()) for x in s["bodies"]])
        g.bemgpu_batch_load.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(P)]
        g.bemgpu_batch_assemble.argtypes = [ctypes.c_void_p]
        g.bemgpu_batch_select.argtypes = [ctypes.c_void_p, ctypes.c_int]
    b.case.solve()  # the resident context, and the solution where the call needs one
    if kind == "solve":
        if case["precision"]:
            b.case.set_precision(case["precision"])
        g.bemgpu_set_interior_reuse(b.case.ctx, 0)
    elif kind == "incident":
        # the mirrored direction has the same in-plane wave vector: the matrices stay
        s["new"] = _Body(case, 180.0 - th, ph, rho, c, amp=(rng.uniform(0.5, 1.5), rng.uniform(-1.0, 1.0)))
        s["new"].problem()
        g.bemgpu_set_incident.argtypes = [ctypes.c_void_p] * 6
        g.bemgpu_solve_rhs.argtypes = [ctypes.c_void_p]
    elif kind == "force9":
        s["rc"] = tuple(rng.uniform(-0.05, 0.05) for _ in range(3))
    elif kind in ("field", "point"):
        n = case.get("count", 1)
        r = np.random.default_rng(seed)
        reach = case["radius"] * case["stretch"]
        v = r.standard_normal((n, 3))
        # outside the body, from a tenth of its radius off the surface to a wavelength away
        s["r"] = v / np.linalg.norm(v, axis=1, keepdims=True) * (reach * r.uniform(1.1, 3.0, (n, 1)))
        if kind == "field":
            g.bemgpu_field.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [api._d, api._d]
            (ax, ay), (bx, by) = lat
            # the grid's points lie in the home cell
            t = np.linalg.solve(np.array([[ax, bx], [ay, by]]), s["r"][:, :2].T)
            s["r"][:, :2] -= (np.array([[ax, bx], [ay, by]]) @ np.round(t)).T
            far = np.linalg.norm(s["r"], axis=1) < 1.08 * reach
            s["r"][far, 2] += 2.2 * reach
    return s


def run(s):
    kind = s["kind"]
    g = api.libs()[1]
    if kind == "dense":
        x = s["b"].copy()
        if g.bemgpu_zgesv(0, s["n"], s["m"], api._p(s["a"].view(np.float64)), api._p(x.view(np.float64))) != 0:
            raise RuntimeError("bemgpu_zgesv failed")
        return x
    if kind == "greens":
        v, dv, _ = api.qpgf(s["qp"], s["r"])
        return [v, dv]
    b = s["body"]
    case = b.case
    if kind == "solve":
        case.solve()
        ctx = case.ctx
        return [_force(ctx)] + _solution(ctx, b.ne)
    if kind == "point":
        _, p, v = case.field("pv_t", s["r"][0], 1)
        return [np.array([p]), v]
    ctx = case.ctx
    if kind == "sweep":
        out = []
        _ok(ctx, g.bemgpu_batch_load(ctx, len(s["probs"]), s["probs"]))
        _ok(ctx, g.bemgpu_batch_assemble(ctx))
        for i in range(len(s["probs"])):
            _ok(ctx, g.bemgpu_batch_select(ctx, i))
            _ok(ctx, g.bemgpu_solve(ctx))
            out.append(_force(ctx))
            sol = _solution(ctx, b.ne)
            out += [np.concatenate([sol[0], sol[1], sol[4], sol[5]]), np.concatenate([sol[2], sol[3], sol[6], sol[7]])]
        return out
    if kind == "incident":
        q = s["new"].problem()
        pw = (ctypes.c_double * 16)(*q.pw)
        _ok(ctx, g.bemgpu_set_incident(ctx, q.Pi, q.dPi, q.p_inc, q.v_inc, pw))
        _ok(ctx, g.bemgpu_solve_rhs(ctx))
        return [_force(ctx)] + _solution(ctx, b.ne)
    if kind == "force9":
        return _force(ctx, 1, s["rc"])
    out = np.zeros((len(s["r"]), 18))
    _ok(ctx, g.bemgpu_field(ctx, 0, 1, len(s["r"]), api._p(s["r"]), api._p(out)))
    return out


def work(case):
    """What a pass cannot do without: FP64 operations (8/3 n^3 of each dense
    factorisation, 8 n^2 of each solve, 36 points of 60 operations per pair of a node
    and a source element) and bytes (inputs once, matrices or results once)."""
    kind = case["kind"]
    if kind == "dense":
        n, m = case["n"], case["count"]
        return {"bytes": 16.0 * n * n + 32.0 * n * m, "flops": 8.0 / 3.0 * n ** 3 + 8.0 * n * n * m}
    if kind == "greens":
        return {"bytes": 92.0 * case["count"], "flops": 2000.0 * case["count"]}
    ne = _elements(case)
    npe = 3 if case["mesh"] == "tri" else 4
    N = npe * ne
    tables, result = 700.0 * ne, 2 * 128.0 * N
    solves = 8.0 * (2 * N) ** 2 + 2 * 8.0 * N * N * 3
    factors = 8.0 / 3.0 * ((2 * N) ** 3 + 2 * N ** 3)
    pairs = 36 * 60.0 * N * ne * 2
    matrices = 16.0 * (2 * 2 * N * N + 4 * N * N + (2 * N) ** 2)
    if kind == "solve":
        return {"bytes": tables + result + matrices, "flops": solves + factors + pairs}
    if kind == "sweep":
        nb = case["count"]
        return {"bytes": nb * (tables + result + matrices), "flops": nb * (solves + factors + pairs)}
    if kind == "incident":
        return {"bytes": tables + result + 16.0 * ((2 * N) ** 2 + 2 * 2 * N * N + 4 * N * N), "flops": solves}
    rule = 7 if case["mesh"] == "tri" else 9
    if kind == "force9":
        return {"bytes": tables + result, "flops": 60.0 * (rule * ne) * (rule * ne + 6144)}
    n = case.get("count", 1)
    return {"bytes": tables + result + 168.0 * n, "flops": 100.0 * n * rule * ne}


def exact(case, seed):
    if case["kind"] == "dense":
        s = prepare(case, seed)
        return np.linalg.solve(s["a"], s["b"].T).T.copy()
    if case["kind"] != "greens":
        # a boundary-value problem's matrices take minutes in numpy
        return None
    # the pure spectral sum, G = i / (2 |cell|) sum_n e^{i a_n . rho + i b_n |z|} / b_n,
    # over the orders with |b_n z| < 38
    s = prepare(case, seed)
    k, kx, ky = s["qp"][:3]
    lat = _lattice(case)
    (g1x, g1y), (g2x, g2y) = _reciprocal(lat)
    cell = abs(lat[0][0] * lat[1][1] - lat[1][0] * lat[0][1])
    r = s["r"]
    v, dv = np.zeros(len(r), np.complex128), np.zeros((len(r), 3), np.complex128)
    az = np.abs(r[:, 2])
    order = np.argsort(az)
    for c0 in range(0, len(r), 64):
        idx = order[c0:c0 + 64]
        amax = 38.0 / az[idx[0]] + k
        gmin = min(math.hypot(g1x, g1y), math.hypot(g2x, g2y)) * 0.8
        m = int(amax / gmin) + 2
        n1, n2 = np.arange(-m, m + 1), np.arange(-m, m + 1)
        ax = -kx + n1[:, None] * g1x + n2[None, :] * g2x
        ay = -ky + n1[:, None] * g1y + n2[None, :] * g2y
        keep = ax * ax + ay * ay < amax * amax
        bn = np.sqrt((k * k - ax * ax - ay * ay)[keep].astype(np.complex128))
        for i in idx:
            x, y, z = r[i]
            e1 = np.exp(1j * n1 * (g1x * x + g1y * y))
            e2 = np.exp(1j * n2 * (g2x * x + g2y * y))
            ph = (e1[:, None] * e2[None, :])[keep] * np.exp(-1j * (kx * x + ky * y))
            prop = bn.imag == 0.0
            t = ph * np.exp(-bn.imag * az[i])
            t[prop] *= np.exp(1j * bn.real[prop] * az[i])
            f = 0.5j / cell
            v[i] = f * np.sum(t / bn)
            dv[i, 0] = f * np.sum(1j * ax[keep] * t / bn)
            dv[i, 1] = f * np.sum(1j * ay[keep] * t / bn)
            dv[i, 2] = f * np.sum(1j * t) * math.copysign(1.0, z)
    return [v, dv]
