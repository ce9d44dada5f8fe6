"""Scenes whose wavelength is read by nothing, by the materials only, or by
the media only: uniform shader values come with the material record, and a
path draws its wavelength only where the scene needs it. All-FP64 build
against the CPU oracle on the same streams (the same paths, so 1e-9: FP64
rounding amplified by distances of 1e2 m)."""
import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu

NODES = [0.4, 0.7, 1.1, 2.0]


def _scene(lib, refl, rough, air):
    s = P.Scene(lib)
    helio = s.mirror((lambda wl, f: 0.5 + 0.2 * wl) if refl else 0.8,
                     (lambda wl, f: 1e-3 * wl) if rough else 2e-3)
    back = s.matte(0.0)
    for i in range(3):
        p = (20.0 * (i - 1), 60.0, 2.0)
        sun, a = W.to_sun(50.0, 180.0), W._unit((-p[0], -p[1], 40.0 - p[2]))
        n = W._unit(tuple(sun[c] + a[c] for c in range(3)))
        s.instance(s.object([(s.rectangle(3, 3), helio, back)]),
                   P.transform_from(W.frame_z_to(n), p))
    rm = s.matte(0.2)
    rcv = s.instance(s.object([(s.rectangle(4, 4), rm, rm)]),
                     P.transform_from(W.frame_z_to((0.0, 0.8, -0.6)), (0.0, 0.0, 40.0)),
                     receiver=P.SSOL_FRONT, sample=0)
    s.set_sun("pillbox", tuple(-c for c in W.to_sun(50.0, 180.0)), 900.0, param=4.65e-3,
              spectrum=s.spectrum(NODES, [1.0, 2.0, 0.5, 0.1]))
    s.atmosphere(s.spectrum(NODES, [1e-3, 5e-4, 2e-3, 1e-4]) if air else 7e-4)
    return s, rcv


@pytest.mark.parametrize("refl,rough,air", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)])
def test_wavelength_dependence_matches_oracle(product, oracle, refl, rough, air):
    res = []
    for lib, opt in ((product, P.options(P.FP64)), (oracle, None)):
        s, rcv = _scene(lib, refl, rough, air)
        e = s.solve(4001, seed=3, options=opt)
        res.append((e.globals(), e.receiver(rcv)))
    for a, b in zip(*res):
        top = max(abs(v[0]) for v in b.values())
        for k in a:
            assert a[k][0] == pytest.approx(b[k][0], rel=1e-9, abs=1e-9 * top), k
