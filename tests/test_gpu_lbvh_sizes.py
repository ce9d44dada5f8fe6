"""The device BVH builder where its path changes: the smallest trees, the most
primitives that one block builds in one launch and one more, trees whose upper
heights share a block, and primitives stacked on one point (no treelet order,
equal Morton codes). A tree finds the closest hits whatever its shape, so a
solve equals the host tree's but for the order of the FP64 sums (1e-10)."""
import random

import pytest

import pyssol as P

pytestmark = pytest.mark.gpu


def _scene(lib, n, stacked):
    """n - 2 scattered mirror triangles (or all about one point) and a
    receiver of two."""
    r = random.Random(n)
    s = P.Scene(lib)
    m, rm = s.mirror(0.9, 2e-3), s.mirror(0.05, 0.0)
    verts, ids = [], []
    for i in range(n - 2):
        c = (0.0, 0.0, 0.02 * i) if stacked else tuple(r.uniform(-30, 30) for _ in range(2)) + (
            r.uniform(0, 3),)
        k = len(verts)
        for _ in range(3):
            verts.append(tuple(c[a] + r.uniform(-2, 2) * (0.1 if a == 2 else 1.0) for a in range(3)))
        ids.append((k, k + 1, k + 2))
    if ids:
        s.instance(s.object([(s.mesh(verts, ids), m, m)]))
    rcv = s.instance(s.object([(s.rectangle(20, 20), rm, rm)]),
                     P.transform_from(((1, 0, 0), (0, -1, 0), (0, 0, -1)), (0.0, 0.0, 40.0)),
                     receiver=P.SSOL_FRONT, sample=0 if ids else 1)
    s.set_sun("pillbox", (0.3, 0.1, -1.0), 1000.0, param=4.65e-3)
    return s, rcv


@pytest.mark.parametrize("n,stacked", [(2, False), (3, False), (4, False), (33, True), (511, False),
                                       (512, False), (512, True), (513, False), (1025, False),
                                       (7001, False)])
@pytest.mark.parametrize("precision", [P.FP32, P.FP64])
def test_device_tree_traces_the_host_trees_paths(product, n, stacked, precision):
    s, rcv = _scene(product, n, stacked)
    got = []
    for bvh in (P.BVH_SAH, P.BVH_LBVH, P.BVH_LBVH):
        e = s.solve(40009, seed=6, options=P.options(precision, bvh=bvh))
        st = e.stats()
        assert st["bvh_nodes"] >= 1 and 1 <= st["bvh_depth"] <= 30
        got.append((e.globals(), e.receiver(rcv), st["bvh_depth"], st["bvh_device"]))
    assert [g[3] for g in got] == [0, 1, 1] and got[1][2] == got[2][2]
    for a in got[1:]:
        for x, y in zip(a[:2], got[0][:2]):
            top = max(abs(v[0]) for v in y.values())
            for k in y:
                assert x[k][0] == pytest.approx(y[k][0], rel=1e-10, abs=1e-10 * top), k
