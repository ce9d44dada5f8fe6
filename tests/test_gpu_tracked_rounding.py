"""The path tracker's kernel traces the paths of the plain one bit for bit, also
where a shader is baked at the vertices: the estimates of a tracked solve are
those of a plain solve of the same realisations but for the order of the FP64
sums (1e5 terms of one sign: 1e-13 leaves room for a hundred times the usual).
One FP32 rounding that differs shows as 1e-11."""
import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 100000])
def test_tracked_is_plain(product, n):
    s = P.Scene(product)
    sun, aim = W.to_sun(50.0, 180.0), (0.0, 0.0, 100.0)
    front = s.mirror(lambda wl, f: 0.8 + 0.001 * f.P[0], 2e-3)
    obj = s.object([(s.rectangle(4, 4), front, s.matte(0.0))])
    for p in W.surround_layout(100):
        a = W._unit(tuple(aim[c] - p[c] for c in range(3)))
        nn = W._unit(tuple(sun[c] + a[c] for c in range(3)))
        s.instance(obj, P.transform_from(W.frame_z_to(nn), p))
    m = s.mirror(0.05, 0.0)
    s.instance(s.object([(W.grid_mesh(s, 12.0, 12.0, 24, 24), m, m)]),
               P.transform_from(P.rotation_pitch_pi(), aim), receiver=P.SSOL_FRONT,
               per_primitive=1, sample=0)
    s.set_sun("pillbox", tuple(-x for x in sun), 900.0, param=4.65e-3)
    a = s.solve(n, seed=1, tracker=(5.0, 5.0)).globals()
    b = s.solve(n, seed=1).globals()
    for k in b:
        assert a[k][0] == pytest.approx(b[k][0], rel=1e-13, abs=1e-13), k
