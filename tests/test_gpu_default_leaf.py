"""The host tree's leaves where the caller leaves them open (two triangles in
scenes of meshes, one primitive with punched surfaces): the same sums as with
one primitive a leaf (1e-10, the order of the sums), in fewer node visits for
meshes and the same for punched surfaces. Plans, and the items of a batch."""
import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu


def _batch(lib, s, opt, n):
    b = P.Batch(lib, [s], opt)
    rng = s.rng(seed=3)
    b.launch(rng, [n])
    return b.finish(rng)[0]


@pytest.mark.parametrize("punched", [False, True])
@pytest.mark.parametrize("batch", [False, True])
def test_default_leaf(product, punched, batch):
    s = (W.beam_down(product, n_helio=60, receiver_cells=5) if punched
         else W.heliostat_field(product, n_helio=37, receiver_cells=7))[0]
    got = []
    for leaf in (0, 1):
        opt = P.options(leaf=leaf, bvh=P.BVH_SAH, count=1)
        e = _batch(product, s, opt, 50021) if batch else s.solve(50021, seed=3, options=opt)
        got.append((e.globals(), e.stats()["node_visits"]))
    (a, na), (b, nb) = got
    for k in b:
        assert a[k][0] == pytest.approx(b[k][0], rel=1e-10, abs=1e-10), k
    assert na == nb if punched else na < nb
