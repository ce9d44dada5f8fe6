"""Pairs of triangles in the host's tree (join_pairs of bvh.cpp) on the CPU:
tests/bvh_host/check_pairs.cpp casts rays in FP32, as the kernels do, through a
tree with leaves of one and through the same tree with its pairs joined. Both must
hit the same triangle at the same distance, whatever the box test rounds away near
the corners of boxes, and on edges that two triangles share."""
import os
import random
import shutil
import subprocess

import pytest

import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "solstice-solver_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pairs") / "check_pairs")
    subprocess.run(["g++", "-O3", "-mfma", "-ffp-contract=off", "-std=c++17", "-I" + CSRC,
                    "-I" + CUDA_INC, os.path.join(ROOT, "tests", "bvh_host", "check_pairs.cpp"),
                    os.path.join(CSRC, "bvh.cpp"), "-o", out, "-lpthread"],
                   check=True, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    return out


def _run(checker, tris, rays=(), extra=0):
    """(rays, those that hit, those that the test of own boxes decides)"""
    text = "%d\n" % len(tris)
    text += "".join(" ".join("%.17g" % c for v in t for c in v) + "\n" for t in tris)
    text += "%d\n" % len(rays) + "".join(" ".join("%.9g" % c for c in r) + "\n" for r in rays)
    p = subprocess.run([checker, str(extra)], input=text, stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300)
    assert p.returncode == 0, p.stdout
    return [int(x) for x in p.stdout.split()[1:]]


def _quad(frame, origin, corners):
    v = [tuple(sum(frame[r][k] * q[k] for k in range(3)) + origin[r] for r in range(3))
         for q in corners]
    return [(v[0], v[2], v[1]), (v[2], v[0], v[3])]


def _field(n, cells, elevation, azimuth, aim=(0.0, 0.0, 100.0)):
    """Triangles of workloads.heliostat_field"""
    sun = W.to_sun(elevation, azimuth)
    tris = []
    for p in W.field_layout(n):
        a = W._unit(tuple(aim[c] - p[c] for c in range(3)))
        frame = W.frame_z_to(W._unit(tuple(sun[c] + a[c] for c in range(3))))
        tris += _quad(frame, p, [(-5, -5, 0), (5, -5, 0), (5, 5, 0), (-5, 5, 0)])
    frame = W.frame_z_to(W._unit((0.0 - aim[0], 350.0 - aim[1], 5.0 - aim[2])))
    for j in range(cells):
        for i in range(cells):
            x, y, d = -6 + 12 * i / cells, -6 + 12 * j / cells, 12 / cells
            tris += _quad(frame, aim, [(x, y, 0), (x + d, y, 0), (x + d, y + d, 0), (x, y + d, 0)])
    return tris


def test_field(checker):
    """Rays at the corners of boxes, a few of them such that the box of the hit
    triangle is missed; the first one came off a mirror of this field."""
    ray = (134.549866, 249.588821, 6.78180456, -0.446441978, -0.835597336, 0.320104957)
    rays, hits, boxed = _run(checker, _field(1000, 64, 58.136079, 196.936615), [ray], 80_000)
    assert rays == 80_001 and hits > rays // 2 and boxed > 0


@pytest.mark.parametrize("cells", [1, 2, 3, 24])
def test_receiver_along_the_axes(checker, cells):
    """Edges shared by triangles whose boxes have their faces in common"""
    frame = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    tris = []
    for j in range(cells):
        for i in range(cells):
            tris += _quad(frame, (i, j, 0.0), [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0)])
    tris += _quad(frame, (-3.0, -3.0, 20.0), [(0, 0, 0), (9, 0, 0), (9, 9, 0), (0, 9, 0)])
    assert _run(checker, tris, extra=100_000)[1] > 10_000


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 33, 2000])
def test_loose_triangles(checker, n):
    rnd = random.Random(n)
    tris = []
    for _ in range(n):
        c = [rnd.uniform(-50, 50) for _ in range(3)]
        tris.append([[x + rnd.uniform(-5, 5) for x in c] for _ in range(3)])
    _run(checker, tris, extra=50_000)
