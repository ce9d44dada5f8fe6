"""BVH leaves of 1 to 9 primitives (both leaves of a node hit, several
primitives in one) and both builders: the traversal finds the same closest
hits whatever the tree, so a solve gives the same sums but for their order
(1e-10). Two and three primitives are the smallest trees."""
import pytest

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu


def _mirror(lib):
    s, h = W.single_mirror(lib)
    return s, h["receiver"]


def _field(lib):
    s, h = W.heliostat_field(lib, n_helio=37, receiver_cells=7)
    return s, h["receiver"]


def _beamdown(lib):
    s, h = W.beam_down(lib, n_helio=60, receiver_cells=5)
    return s, h["receiver"]


@pytest.mark.parametrize("make", [_mirror, _field, _beamdown])
@pytest.mark.parametrize("precision", [P.FP32, P.FP64])
def test_leaf_sizes_trace_the_same_paths(product, make, precision):
    s, rcv = make(product)
    ref = None
    for leaf, bvh in ((1, P.BVH_SAH), (2, P.BVH_SAH), (4, P.BVH_SAH), (9, P.BVH_SAH),
                      (1, P.BVH_LBVH)):
        e = s.solve(60011, seed=8, options=P.options(precision, leaf=leaf, bvh=bvh))
        got = [e.globals(), e.receiver(rcv)]
        if ref is None:
            ref = got
            continue
        for a, b in zip(got, ref):
            top = max(abs(v[0]) for v in b.values())
            for k in b:
                assert a[k][0] == pytest.approx(b[k][0], rel=1e-10, abs=1e-10 * top), (leaf, k)
