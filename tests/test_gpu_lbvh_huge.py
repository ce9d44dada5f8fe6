"""The device BVH builder on a scene so large that the SAH costs of whole
subtrees overflow FP32 (60,000 overlapping triangles 1e17 wide: 60,000 x 1e34 is
above 3.4e38, while the area of the root, 1e35, is not). No order of a treelet is
better than another there, and the tree must stay the tree it was: the estimates
are the host tree's but for the order of the FP64 sums (1e-10)."""
import random

import pytest

import pyssol as P

pytestmark = pytest.mark.gpu


def test_overflowing_costs_leave_the_tree_whole(product):
    r = random.Random(4)
    s = P.Scene(product)
    m, rm = s.mirror(0.9, 0.0), s.mirror(0.05, 0.0)
    verts, ids = [], []
    for i in range(60000):
        c = (r.uniform(-3e16, 3e16), r.uniform(-3e16, 3e16), r.uniform(-3e16, 3e16))
        for _ in range(3):
            verts.append((c[0] + r.uniform(-1e17, 1e17), c[1] + r.uniform(-1e17, 1e17),
                          c[2] + r.uniform(-1e15, 1e15)))
        ids.append((3 * i, 3 * i + 1, 3 * i + 2))
    s.instance(s.object([(s.mesh(verts, ids), m, m)]))
    rcv = s.instance(s.object([(s.rectangle(2e17, 2e17), rm, rm)]),
                     P.transform_from(((1, 0, 0), (0, -1, 0), (0, 0, -1)), (0.0, 0.0, 1e17)),
                     receiver=P.SSOL_FRONT, sample=0)
    s.set_sun("pillbox", (0.3, 0.1, -1.0), 1000.0, param=4.65e-3)
    got = []
    for bvh in (P.BVH_SAH, P.BVH_LBVH):
        e = s.solve(4001, seed=6, options=P.options(P.FP64, bvh=bvh))
        st = e.stats()
        assert st["bvh_device"] == (bvh == P.BVH_LBVH) and 1 <= st["bvh_depth"] <= 30
        got.append((e.globals(), e.receiver(rcv)))
    for x, y in zip(got[1], got[0]):
        top = max(abs(v[0]) for v in y.values())
        for k in y:
            assert x[k][0] == pytest.approx(y[k][0], rel=1e-10, abs=1e-10 * top), k
