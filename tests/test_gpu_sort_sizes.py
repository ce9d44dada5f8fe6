"""The presort where its sizes change: the smallest sorted launch and the one
below, counts that leave a ragged last segment and tile, scenes whose sampled
primitives just fill the histogram's bins, exceed them (several neighbours to
a bin), or belong to one instance. The same realisations launched in pieces
below the threshold run in id order: the same paths, so the same sums but for
their order (1e-10, as FP64 sums of 1e6 terms)."""
import ctypes as C

import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu

SORT_MIN = 200000


def _sheet(lib, nx, ny, copies):
    s = P.Scene(lib)
    m, r = s.mirror(0.9, 2e-3), s.mirror(0.05, 0.0)
    mesh = W.grid_mesh(s, 10.0, 10.0, nx, ny)
    obj = s.object([(mesh, m, m)])
    for i in range(copies):
        s.instance(obj, P.transform_from(None, (12.0 * i, 0.0, 0.0)))
    rcv = s.instance(s.object([(s.rectangle(4, 4), r, r)]),
                     P.transform_from(((1, 0, 0), (0, -1, 0), (0, 0, -1)), (0.0, 0.0, 20.0)),
                     receiver=P.SSOL_FRONT, sample=0)
    s.set_sun("pillbox", (0.05, 0.0, -1.0), 1000.0, param=4.65e-3)
    return s, rcv


def _solve(lib, s, n, step):
    plan, est, rng = C.c_void_p(), C.c_void_p(), s.rng(seed=4)
    lib.call("ssol_b200_plan_create", s.scn, None, C.byref(plan))
    for first in range(0, n, step):
        lib.call("ssol_b200_plan_launch", plan, rng, first, min(step, n - first), None)
    lib.call("ssol_b200_plan_finish", plan, rng, n, 0, None, C.byref(est))
    lib.raw("ssol_b200_plan_ref_put", plan)
    return P.Estimator(s, est, P.RES_OK)


def _scene(lib, kind):
    if kind == "field2":
        s, h = W.heliostat_field(lib, n_helio=2, receiver_cells=4)
        return s, h["receiver"]
    if kind == "field700":
        s, h = W.heliostat_field(lib, n_helio=700, receiver_cells=4)
        return s, h["receiver"]
    return _sheet(lib, *{"bins": (64, 48, 2), "over": (64, 48, 3), "far over": (100, 150, 4),
                         "one": (32, 16, 1)}[kind])


@pytest.mark.parametrize("kind", ["field2", "field700", "bins", "over", "far over", "one"])
@pytest.mark.parametrize("n", [SORT_MIN - 1, SORT_MIN, SORT_MIN + 33, 5 * SORT_MIN + 12345])
def test_sorted_equals_id_order(product, kind, n):
    s, rcv = _scene(product, kind)
    a, b = _solve(product, s, n, n), _solve(product, s, n, SORT_MIN - 1)
    for x, y in ((a.globals(), b.globals()), (a.receiver(rcv), b.receiver(rcv))):
        top = max(abs(v[0]) for v in y.values())
        for k in x:
            assert x[k][0] == pytest.approx(y[k][0], rel=1e-10, abs=1e-10 * top), k
            assert x[k][1] == pytest.approx(y[k][1], rel=1e-9, abs=1e-9 * top * top), k
    assert a.count("realisation_count") == b.count("realisation_count") == n
