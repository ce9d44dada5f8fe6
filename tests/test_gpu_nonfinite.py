"""Weights that are not finite stay in the slots of the paths that carry them:
they are added by reductions of their own, not through the warp's tiles, where
a zero times infinity would reach the other sums. One heliostat with an infinite
reflectivity beside a sound one, sampled by the same warps; all-FP64 build
against the oracle (1e-9, as in the commit's test). A reflectivity of NaN is
refused before any launch: the shader's values differ between two evaluations."""
import math

import pytest

import pyssol as P

pytestmark = pytest.mark.gpu


def _solve(lib, bad, opt):
    s = P.Scene(lib)
    good, broken = s.mirror(0.9, 0.0), s.mirror(lambda wl, f: bad, 0.0)
    shape = s.rectangle(4, 4)
    a = s.instance(s.object([(shape, good, good)]), P.transform_from(None, (-5.0, 0.0, 0.0)))
    b = s.instance(s.object([(shape, broken, broken)]), P.transform_from(None, (5.0, 0.0, 0.0)))
    rm = s.matte(0.0)
    rcv = s.instance(s.object([(s.rectangle(9, 3), rm, rm)]),
                     P.transform_from(((1, 0, 0), (0, -1, 0), (0, 0, -1)), (0.0, 6.0, 10.0)),
                     receiver=P.SSOL_FRONT, sample=0)
    s.set_sun("pillbox", (0.0, 0.6, -1.0), 1000.0, param=4.65e-3)
    e = s.solve(4099, seed=2, options=opt)
    return (e.globals(), e.sampled_x_receiver(a, rcv), e.sampled_x_receiver(b, rcv),
            e.receiver(rcv), e.sampled(a), e.sampled(b))


def test_nan_shader_is_refused(product):
    with pytest.raises(P.SsolError):
        _solve(product, math.nan, P.options(P.FP64))


@pytest.mark.parametrize("bad", [math.inf])
def test_broken_heliostat_keeps_to_itself(product, oracle, bad):
    x, y = _solve(product, bad, P.options(P.FP64)), _solve(oracle, bad, None)
    for p, q in zip(x, y):
        for k in q:
            if k == "nb_samples":
                assert p[k] == q[k]
                continue
            u, v = p[k][0], q[k][0]
            if math.isfinite(v):
                assert u == pytest.approx(v, rel=1e-9, abs=1e-6), k
            else:
                assert not math.isfinite(u), k
    assert math.isfinite(x[1]["incoming_flux"][0]) and x[1]["incoming_flux"][0] > 0
    assert math.isfinite(x[1]["absorbed_flux"][0])
