"""Adjoint passes in the coherent order (from 2e5 realisations) against the
same realisations in pieces that run in id order. The absorbed power, its
gradient and the map are means over realisations, so a call is the weighted
mean of its pieces; FP64 sums in another order (1e-10). Counts that leave a
ragged segment; one heliostat (id order whatever the count), two, many."""
import numpy as np
import pytest

import adjoint as A
import workloads as W

pytestmark = pytest.mark.gpu


def _run(s, h, n, position):
    rng = type(s).rng
    s.rng = lambda seed=0: rng(s, seed, position)
    try:
        r = A.solve_adjoint(s, h["heliostats"], h["receiver"], (-6, -6), (6, 6), 16, 16, 1e3, n,
                            seed=2, want_map=True)
    finally:
        del s.rng
    return np.concatenate([[r["absorbed"]], r["d_absorbed"], r["map"]]), r["hits"]


@pytest.mark.parametrize("helios", [1, 2, 90])
@pytest.mark.parametrize("n", [200000, 200000 + 31, 777777])
def test_sorted_adjoint_is_the_mean_of_its_pieces(product, helios, n):
    s, h = W.heliostat_field(product, n_helio=helios, receiver_cells=2)
    whole, hits = _run(s, h, n, 0)
    mean, count, step = 0.0, 0, 150000
    for first in range(0, n, step):
        k = min(step, n - first)
        v, c = _run(s, h, k, first)
        mean, count = mean + v * (k / n), count + c
    assert hits == count
    assert np.linalg.norm(whole - mean) <= 1e-10 * np.linalg.norm(mean)
