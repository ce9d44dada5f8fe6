"""Buie's rejection loop decides most attempts in FP32 and the closest ones in
FP64: every accepted angle must be the one the FP64 comparison alone accepts.
The sun end of each tracked path lies 1000 m along the sampled direction; a
different decision on any attempt moves it by metres, FP64 rounding by 1e-9."""
import pytest

import pyssol as P

pytestmark = pytest.mark.gpu


def _ends(lib, csr, n, opt):
    s = P.Scene(lib)
    m = s.matte(0.5)
    s.instance(s.object([(s.rectangle(5, 5), m, m)]), receiver=P.SSOL_FRONT)
    s.set_sun("buie", (0.2, -0.1, -1.0), 1000.0, param=csr)
    e = s.solve(n, seed=21, options=opt, tracker=(1000.0, 1.0))
    return [verts[0][0] for _, verts in e.paths()]


@pytest.mark.parametrize("csr", [0.002, 0.02, 0.1, 0.3, 0.7])
def test_every_angle_is_the_oracles(product, oracle, csr):
    n = 12007
    a = _ends(product, csr, n, P.options(P.FP64))
    b = _ends(oracle, csr, n, None)
    assert len(a) == len(b) == n
    worst = max(max(abs(x - y) for x, y in zip(p, q)) for p, q in zip(a, b))
    assert worst < 1e-6
