"""The warp's commit: paths of one sampled instance are summed through the
warp's tiles, the others by reductions of their own. Sizes where the split
changes: one lane, a partial warp, several warps; one heliostat (every lane
in one group), a few (groups and single lanes mixed), many (single lanes).
All-FP64 build against the CPU oracle on the same streams: the same paths, so
the estimates differ by the rounding of FP64 path arithmetic only (1e-16 per
operation, amplified by distances of 1e3 m over edges of 1 m: below 1e-9)."""
import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu
REL = 1e-9


def _close(a, b, scale, what):
    assert a[0] == pytest.approx(b[0], rel=REL, abs=REL * scale), what
    assert a[1] == pytest.approx(b[1], rel=REL, abs=REL * scale * scale), what


@pytest.mark.parametrize("helios", [1, 2, 7, 60])
@pytest.mark.parametrize("n", [1, 3, 31, 33, 257, 9001])
def test_commit_matches_oracle(product, oracle, helios, n):
    got = []
    for lib, opt in ((product, P.options(P.FP64)), (oracle, None)):
        s, h = W.heliostat_field(lib, n_helio=helios, receiver_cells=3)
        e = s.solve(n, seed=5, options=opt)
        got.append((s, h, e))
    (_, ha, ea), (_, hb, eb) = got
    ga, gb = ea.globals(), eb.globals()
    top = 900.0 * 100.0 * helios
    for k in ga:
        _close(ga[k], gb[k], top, k)
    ra, rb = ea.receiver(ha["receiver"]), eb.receiver(hb["receiver"])
    for k in ra:
        _close(ra[k], rb[k], top, k)
    pa = ea.primitives(ha["receiver"], ha["receiver_shape"])
    pb = eb.primitives(hb["receiver"], hb["receiver_shape"])
    for x, y in zip(pa, pb):
        for k in x:
            _close(x[k], y[k], top, k)
    total = 0
    for ia, ib in zip(ha["heliostats"], hb["heliostats"]):
        xa, xb = ea.sampled(ia), eb.sampled(ib)
        assert xa["nb_samples"] == xb["nb_samples"]
        total += xa["nb_samples"]
        _close(xa["cos_factor"], xb["cos_factor"], 1.0, "cos")
        _close(xa["shadowed"], xb["shadowed"], top, "shadowed")
        if xa["nb_samples"]:
            ya = ea.sampled_x_receiver(ia, ha["receiver"])
            yb = eb.sampled_x_receiver(ib, hb["receiver"])
            for k in ya:
                _close(ya[k], yb[k], top, k)
    assert total == n


@pytest.mark.parametrize("budgets", [(1, 40, 7), (3000, 1, 5000, 33)])
def test_batch_items_in_one_warp(product, budgets):
    """Warps that straddle items key their tiles by item: each item's sums
    are those of its own solve (1e-10: FP64 sums in another order)."""
    scenes = [W.heliostat_field(product, n_helio=1 + 3 * i, receiver_cells=2, dni=500.0 + 50 * i)
              for i in range(len(budgets))]
    b = P.Batch(product, [s for s, _ in scenes], P.options(P.FP64))
    rng = scenes[0][0].rng(seed=9)
    b.reset()
    b.launch(rng, budgets)
    for (s, h), n, e in zip(scenes, budgets, b.finish(rng)):
        ref = s.solve(n, seed=9, options=P.options(P.FP64))
        for k, v in e.globals().items():
            assert v[0] == pytest.approx(ref.globals()[k][0], rel=1e-10, abs=1e-9), k
        x, y = e.receiver(h["receiver"]), ref.receiver(h["receiver"])
        for k in x:
            assert x[k][0] == pytest.approx(y[k][0], rel=1e-10, abs=1e-9), k
    b.close()
