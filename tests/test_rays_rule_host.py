"""Where the ionizing rays march without clamps (csrc/nb_rays_rule.h, compiled here as plain C++): at the
rule's limit every sample's corners lie inside the grid, whatever the last bit of the approximate
reciprocals.  The kernel's index arithmetic is restated in numpy float32; no GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
f = np.float32


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text('#include <cstdlib>\n#include "nb_rays_rule.h"\n'
                                "int main(int, char** v) { return nb_march_unclamped(atoi(v[1]), atoi(v[2]), atoi(v[3]), "
                                "atoi(v[4]), strtof(v[5], 0), strtof(v[6], 0)) ? 10 : 20; }\n")
    exe = str(d / "rule")
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "nebulaviewer_gb300", "csrc"), str(d / "rule.cpp"), "-o",
                    exe], check=True)

    def ask(shape, nsteps, dr, dx):
        rc = subprocess.run([exe, *(str(n) for n in shape), str(nsteps), repr(float(dr)), repr(float(dx))]).returncode
        assert rc in (10, 20)
        return rc == 10
    return ask


def outside_corners(shape, nsteps, dr, dx, away, rays, rng):
    """samples of the unclamped part whose corners leave the grid, over rays from a star `away` cells from
    the box to points in it"""
    dr, dx = f(dr), f(dx)
    bmax = [f(n) * dx for n in shape]
    bad = seen = 0
    for _ in range(rays):
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        target = np.array([rng.uniform(0, n) for n in shape]) * float(dx)
        o = (target + u * away * float(dx)).astype(np.float32)
        d = target - o.astype(np.float64)
        d = (d / np.linalg.norm(d)).astype(np.float32)
        with np.errstate(all="ignore"):
            w = (f(1) / d).astype(np.float32)
            w = (w * (1 + f(2.0 ** -23) * rng.integers(-1, 2, 3).astype(np.float32))).astype(np.float32)
            i0, i1 = f(0), f(1e9)
            for a in range(3):
                ta, tb = (dx - o[a]) * w[a], ((bmax[a] - dx) - o[a]) * w[a]
                i0, i1 = max(i0, min(ta, tb)), min(i1, max(ta, tb))
            inv = f(f(1) / dr * (1 + f(2.0 ** -23) * f(rng.integers(-1, 2))))
            in0, in1 = f(i0 * inv), min(f(i1 * inv), f(nsteps))
        if not in1 > in0:
            continue
        first = int(np.floor(float(in0)))
        n = np.arange(max(first - 2, 0), min(int(float(in1)) + 3, nsteps), dtype=np.float64) + 0.5
        nf = n.astype(np.float32)
        nf = nf[(nf >= in0) & (nf < in1)]
        r = (nf * dr).astype(np.float32)
        for a in range(3):
            g = ((o[a] + d[a] * r).astype(np.float32) / dx - f(0.5)).astype(np.float32)
            k = np.floor(g)
            bad += int(((k < 0) | (k > shape[a] - 2)).sum())
        seen += nf.size
    return bad, seen


@pytest.mark.parametrize("shape", ((4, 4, 4), (5, 64, 200), (4, 6, 65536), (96, 96, 96)))
def test_corners_stay_inside_at_the_limit(rule, shape):
    rng = np.random.default_rng(sum(shape))
    for dx in (1.0 / 64, 0.01, 3e-4):
        for step in (1.0, 0.5):
            dr = f(f(dx) * f(step))
            nsteps = int(2 ** 18 / step * 0.9999)
            assert rule(shape, nsteps, dr, dx)
            bad, seen = outside_corners(shape, nsteps, dr, dx, 2 ** 18 * 0.999 - 1.5 * max(shape), 600, rng)
            assert seen > 50 and bad == 0


def test_longer_ways_are_clamped(rule):
    for dx in (1.0 / 64, 0.01):
        for step in (1.0, 0.5):
            assert not rule((64, 64, 64), int(2 ** 18 / step * 1.001), f(dx) * f(step), dx)
    # what the limit keeps out: a star 4 million cells away, within the limit on the samples alone
    assert not rule((64, 64, 64), 1 << 22, 0.01, 0.01)
    assert outside_corners((64, 64, 64), 1 << 22, 0.01, 0.01, 4.1e6, 150, np.random.default_rng(1))[0] > 0


def test_other_limits(rule):
    assert rule((64, 64, 64), 200, 1 / 64, 1 / 64)
    for shape in ((3, 64, 64), (64, 3, 64), (64, 64, 3), (65537, 4, 4), (2048, 2048, 512)):
        assert not rule(shape, 200, 1 / 64, 1 / 64)
    assert not rule((64, 64, 64), (1 << 22) + 1, 1e-6, 1 / 64)
    assert not rule((64, 64, 64), 200, 1e-13, 1e-13) and not rule((64, 64, 64), 200, 1e12, 1e12)
    assert not rule((64, 64, 64), 200, float("inf"), 1 / 64) and not rule((64, 64, 64), 200, float("nan"), 1 / 64)
