"""A leaf size that the caller gives is the host tree's: the default builder of
the renderers and the adjoint then visits the nodes of the host's tree of that
size (counted exactly), and those of the device's tree only without one, and in
scenes of 449 primitives or more, below which the host builds its tree sooner."""
import pytest
import torch

import adjoint as A
import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,helio,cells", [(0, 200, 9), (1, 200, 9), (2, 200, 9), (4, 200, 9),
                                              (0, 161, 8), (0, 160, 8), (0, 2, 1)])
def test_default_builder(product, leaf, helio, cells):
    s, h = W.heliostat_field(product, n_helio=helio, receiver_cells=cells)
    cam = s.camera((0.0, -60.0, 170.0), (0.0, 280.0, 0.0), (0.0, 0.0, 1.0), fov=1.3, ratio=1.0)
    px = torch.empty((40, 40, 3), dtype=torch.float64, device="cuda")

    def visits(bvh):
        opt = P.options(leaf=leaf, bvh=bvh)
        draft = s.draw_device("draft", cam, 40, 40, 4, px.data_ptr(), options=opt).node_visits
        r = A.solve_adjoint(s, h["heliostats"], h["receiver"], (-6.0, -6.0), (6.0, 6.0), 9, 9,
                            1e3, 20011, seed=3, options=opt)
        return draft, r["counters"]["node_visits"]

    auto, sah, lbvh = (visits(b) for b in (P.BVH_AUTO, P.BVH_SAH, P.BVH_LBVH))
    assert helio < 100 or all(a != b for a, b in zip(sah, lbvh)), (sah, lbvh)
    assert auto == (sah if leaf or 2 * helio + 2 * cells * cells < 449 else lbvh)
