"""Launches in the coherent order against the same realisations in pieces that
are too small for it and run in id order: the same paths, so the same sums but
for their order (FP64 sums of up to 1.7e7 terms of one sign: 1e-10). The
thresholds are read from the source, so that a change of theirs leaves the pieces
below them. Launches of several chunks, scenes of quadrics and dielectrics,
batches whose items have more sampled primitives than the sort has bins, and the
adjoint's spillage gradient."""
import ctypes as C
import os
import re

import numpy as np
import pytest
import torch

import adjoint as A
import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "csrc")


def _constant(name, file="kernels_device.cuh"):
    with open(os.path.join(CSRC, file)) as f:
        value = re.search(r"\b%s = (\d+)(?:ull)?(?: << (\d+))?[,;]" % name, f.read())
    return int(value[1]) << int(value[2] or 0)


SORT_MIN, SORT_MIN_QUADRIC = _constant("SORT_MIN"), _constant("SORT_MIN_QUADRIC")
SORT_MAX_BINS, BATCH_SORT_MIN = _constant("SORT_MAX_BINS"), _constant("BATCH_SORT_MIN", "solve.cpp")


def _tallies(lib, s, n, step):
    h = C.c_void_p()
    lib.call("ssol_b200_plan_create", s.scn, None, C.byref(h))
    try:
        rng = s.rng(seed=11)
        for first in range(0, n, step):
            lib.call("ssol_b200_plan_launch", h, rng, first, min(step, n - first), None)
        torch.cuda.synchronize()
        sums, counts = P.plan_tallies(lib, h)
        return torch.as_tensor(sums, device="cuda").clone(), torch.as_tensor(counts, device="cuda").clone()
    finally:
        lib.raw("ssol_b200_plan_ref_put", h)


def _same(a, b, nsampled):
    (sa, ca), (sb, cb) = a, b
    assert bool((ca[:nsampled] == cb[:nsampled]).all())
    assert float(((sa - sb).abs() / sb.abs().clamp(min=1e-300)).max()) < 1e-10


def test_two_chunks(product):
    s, h = W.heliostat_field(product, n_helio=700, receiver_cells=32)
    n = (1 << 24) + 12345
    _same(_tallies(product, s, n, n), _tallies(product, s, n, SORT_MIN - 1), 700)


@pytest.mark.parametrize("n", [SORT_MIN_QUADRIC - 1, SORT_MIN_QUADRIC, SORT_MIN_QUADRIC + 33,
                               2 * SORT_MIN_QUADRIC + 12345])
def test_quadrics(product, n):
    s, h = W.beam_down(product, n_helio=60, receiver_cells=5)
    _same(_tallies(product, s, n, n), _tallies(product, s, n, SORT_MIN_QUADRIC - 1), 60)


def test_dielectrics(product):
    s, _ = W.heliostat_field(product, n_helio=60, receiver_cells=5)
    pane = s.thin_dielectric(s.medium(1e-4, 1.0), s.medium(20.0, 1.5), 5e-3)
    s.instance(s.object([(s.rectangle(10, 10), pane, pane)]),
               P.transform_from(((1, 0, 0), (0, 0, -1), (0, 1, 0)), (0.0, 5.0, 100.0)), sample=0)
    n = SORT_MIN_QUADRIC + 77
    _same(_tallies(product, s, n, n), _tallies(product, s, n, SORT_MIN_QUADRIC - 1), 60)


def _sheet(lib, nx, ny, copies):
    s = P.Scene(lib)
    m, r = s.mirror(0.9, 2e-3), s.mirror(0.05, 0.0)
    obj = s.object([(W.grid_mesh(s, 10.0, 10.0, nx, ny), m, m)])
    for i in range(copies):
        s.instance(obj, P.transform_from(None, (12.0 * i, 0.0, 0.0)))
    s.instance(s.object([(s.rectangle(4, 4), r, r)]),
               P.transform_from(((1, 0, 0), (0, -1, 0), (0, 0, -1)), (0.0, 0.0, 20.0)),
               receiver=P.SSOL_FRONT, sample=0)
    s.set_sun("pillbox", (0.05, 0.0, -1.0), 1000.0, param=4.65e-3)
    return s


def test_batch_of_more_primitives_than_bins(product):
    """Items of 12286, 12288, 18432 and 120000 sampled primitives: bins of one,
    two and sixteen neighbours, and bins that stay empty between the items'."""
    assert SORT_MAX_BINS == 12288
    scenes = [_sheet(product, *k) for k in ((6143, 1, 1), (64, 48, 2), (64, 48, 3), (100, 150, 4),
                                            (64, 48, 3))]
    budgets = [BATCH_SORT_MIN // 4 + 1, 200003, 500009, BATCH_SORT_MIN // 2 + 77, 0]
    assert sum(budgets) >= BATCH_SORT_MIN
    got = []
    for parts in (1, 4):
        b = P.Batch(product, scenes)
        rng = scenes[0].rng(seed=5)
        for k in range(parts):
            part = [n * (k + 1) // parts - n * k // parts for n in budgets]
            assert parts == 1 or sum(part) < BATCH_SORT_MIN
            b.launch(rng, part)
        got.append([(e.globals(), e.count("realisation_count"), e.count("failed_count"))
                    for e in b.finish(rng)[:4]])
        b.close()
    for (a, *na), (b, *nb), n in zip(*got, budgets):
        assert na == nb and sum(na) == n
        for k in b:
            assert a[k][0] == pytest.approx(b[k][0], rel=1e-10, abs=1e-10), k


def test_spillage_gradient(product):
    """d/d(angle) of sum (M - T)^2 is 2 sum (M - T) dM: for a target T that is
    1e10 times the map and more, -2 T sum dM to 1e-10, the mean of its pieces' as dM is."""
    s, h = W.heliostat_field(product, n_helio=90, receiver_cells=2)

    def run(n, position):
        make = type(s).rng
        s.rng = lambda seed=0: make(s, seed, position)
        try:
            r = A.solve_adjoint(s, h["heliostats"], h["receiver"], (-6, -6), (6, 6), 16, 16, 1e16,
                                n, seed=2, want_map=True)
        finally:
            del s.rng
        assert max(r["map"]) < 1e6
        return np.array(r["d_spillage"])

    n, step = 3 * SORT_MIN + 17, SORT_MIN - 1
    whole = run(n, 0)
    mean = sum(run(min(step, n - f), f) * (min(step, n - f) / n) for f in range(0, n, step))
    assert np.linalg.norm(whole) > 0
    assert np.linalg.norm(whole - mean) <= 1e-9 * np.linalg.norm(mean)
