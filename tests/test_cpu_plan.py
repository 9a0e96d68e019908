"""The host code that plans the split of the periodic domain (bem_smooth_plan and
bem_smooth_plan_field in the built library, run from a small program, no GPU): the
images taken out are whole shells of the nearest lattice points, the cut clears the ball,
the degree is the one that the truncation rule of test_cpu_smooth.py gives, and a plan
for field points far away is declined at little cost.

Time: a declined plan looks at 41 lattice points kept with the problem; a list of all out
to the points took 24 to 150 ms a call on one core, the bound is 1 ms on average."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_cpu_smooth import _degree

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "bem3_aw_qd2_b200", "lib")
CUDA = "/usr/local/cuda/include"
PROGRAM = r"""
#include <chrono>
#include <cmath>
#include <cstdio>
#include <vector>
#include "bem_smooth.h"
#include "bem_lattice.h"
int main() {
  double p[8], r, st, Rx, n;
  int ne;
  // lattice and wave numbers, a body of six point-like elements on the axes, ne of them in turn
  while (scanf("%lf %lf %lf %lf %lf %lf %lf %lf %lf %lf %d %lf %lf", p, p + 1, p + 2, p + 3, p + 4, p + 5, p + 6, p + 7, &r,
               &st, &ne, &Rx, &n) == 13) {
    bem_qp q;
    bem_qp_prepare(p, &q);
    std::vector<double> cr(72, 0.0);
    std::vector<int> npe(6, 4), sid;
    for (int i = 0; i < 6; ++i) cr[12 * i + 4 * (i / 2)] = (i % 2 ? -r : r) * (i / 2 == 2 ? st : 1.0);
    for (int i = 0; i < ne; ++i) sid.push_back(i % 6 + 1);
    bem_smooth S, F;
    bem_smooth_plan(&S, &q, cr.data(), npe.data(), sid.data(), ne);
    printf("%d %.17g %d %d %.17g", S.on, S.R0, S.on ? S.lmax : 0, S.on ? S.nimg : 0, S.on ? S.cut + S.rho : 0.0);
    for (int i = 0; S.on && i < S.nimg; ++i) printf(" %d %d", S.l1[i], S.l2[i]);
    double ms = 0.0;
    if (S.on && Rx > 0.0) {
      const auto t = std::chrono::steady_clock::now();
      for (int i = 0; i < 20; ++i) bem_smooth_plan_field(&F, &S, &q, Rx, n, 9.0 * ne, 1e300);
      ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count() / 20.0;
    }
    printf("\n%d %.3f\n", S.on && Rx > 0.0 ? F.on : 0, ms);
  }
}
"""
LATTICES = {"square": ((1.0, 0.0), (0.0, 1.0)), "triangular": ((1.0, 0.0), (0.5, 0.75 ** 0.5)),
            "oblique": ((1.0, 0.0), (0.3, 0.9)), "skewed": ((1.0, 0.0), (7.3, 0.8)), "long": ((1.0, 0.0), (0.0, 6.0))}


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = os.path.join(LIB, "libbemgpu.so")
    if not (shutil.which("g++") and os.path.exists(so) and os.path.exists(CUDA)):
        pytest.skip("needs g++, the CUDA headers and the built library")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CUDA, "-I" + os.path.join(ROOT, "bem3_aw_qd2_b200", "csrc"),
                    str(d / "plan.cpp"), so, "-Wl,-rpath," + LIB, "-o", str(d / "plan")], check=True)

    def run(cases):
        k, lines = 2.0 * math.pi, []
        for lat, a, r, st, ne, Rx, n in cases:
            kx, ky = 0.24 * k, 0.18 * k
            v = [k, kx, ky, math.sqrt(k * k - kx * kx - ky * ky)] + [a * x for d in LATTICES[lat] for x in d]
            lines.append(" ".join("%.17g" % x for x in v + [r, st]) + " %d %.17g %.17g" % (ne, Rx, n))
        out = subprocess.run([str(d / "plan")], input="\n".join(lines), capture_output=True, text=True, check=True)
        rows = out.stdout.split("\n")
        return [(rows[2 * i].split(), rows[2 * i + 1].split()) for i in range(len(cases))]

    return run


def test_images_are_whole_shells(plan):
    cases = [(lat, a, f * a, st, ne, 0.0, 0.0) for lat in LATTICES for a in (0.7, 1.0, 3.3) for f in (0.15, 0.3)
             for st in (1.0, 1.5) for ne in (24, 600)]
    on = 0
    for (lat, a, r, st, _, _, _), (row, _) in zip(cases, plan(cases)):
        if row[0] == "0":
            continue
        on += 1
        R0, lmax, nimg, cut = float(row[1]), int(row[2]), int(row[3]), float(row[4])
        got = {(int(x), int(y)) for x, y in zip(row[5::2], row[6::2])}
        assert abs(R0 - r * max(1.0, st)) < 1e-9 and len(got) == nimg and cut > 2.1 * R0
        (ax, ay), (bx, by) = LATTICES[lat]
        i, j = (v.ravel() for v in np.meshgrid(np.arange(-60, 61), np.arange(-60, 61)))
        d = a * np.hypot(i * ax + j * bx, i * ay + j * by)
        assert abs(np.min(d[d > cut * (1 - 1e-9)]) - cut) < 1e-9 * cut
        assert got == {(int(x), int(y)) for x, y, z in zip(i, j, d) if z < cut * (1 - 1e-9)}
        if cut < 4.0:  # (beyond, the sizes that the plan compares are upper bounds)
            assert lmax == _degree(2.0 * math.pi, R0, cut - R0, 12.0 * R0)
    assert on > len(cases) // 2


@pytest.mark.parametrize("lat", sorted(LATTICES))
def test_far_points_are_declined_quickly(plan, lat):
    cases = [(lat, 0.8, 0.24, 1.0, 216, Rx, 2000.0) for Rx in (10.0, 30.0, 60.0, 150.0)]
    for row, (on, ms) in plan(cases):
        assert on == "0" and float(ms) < 1.0, (row[:5], ms)
