"""What a ray meets does not depend on the tree. The box test rounds, so a
triangle hit at a corner of its box can have the box missed by an ulp; whether
it is then found must not depend on the leaf that holds it. About one path in
1e9 of the field is such a one: the two suns here have one each among their
first 1e8 paths (3e-8 of the estimates, hundreds of times the tolerance). The
sums of 1e8 positive FP64 terms in two orders differ by about sqrt(1e8) x
2^-53 = 1e-12 of their value: 1e-10 leaves room for a factor of a hundred."""
import ctypes as C

import pytest
import torch

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu
CELLS, PATHS = 64, 100_000_000


def _trace(lib, s, key, **kw):
    h = C.c_void_p()
    opt = P.options(**kw)
    lib.call("ssol_b200_plan_create", s.scn, C.byref(opt), C.byref(h))
    try:
        lib.call("ssol_b200_plan_launch", h, s.rng(seed=key), 0, PATHS, None)
        sums, _ = P.plan_tallies(lib, h)
        torch.cuda.synchronize()
        return torch.as_tensor(sums, device="cuda").clone()
    finally:
        lib.raw("ssol_b200_plan_ref_put", h)


def _worst(a, b):
    return float(((a - b).abs() / b.abs().clamp(min=1e-300)).max())


@pytest.mark.parametrize("elevation,azimuth,dni,key", [
    (43.67955566060546, 184.19941100288258, 648.9833655313992, 721134112221),
    (47.746183107270284, 154.54201544719152, 705.5378800463839, 70579143265)])
def test_leaves_and_builders_trace_the_same_paths(product, elevation, azimuth, dni, key):
    s, _ = W.heliostat_field(product, n_helio=1000, elevation=elevation, azimuth=azimuth,
                             dni=dni, receiver_cells=CELLS)
    one = _trace(product, s, key, leaf=1, bvh=P.BVH_SAH)
    assert _worst(_trace(product, s, key, bvh=P.BVH_SAH), one) < 1e-10
    # A hit on the edge of two triangles is one of either's, as the tree has
    # them: the flux map (the last sums) may have it in the neighbour
    flux = 2 * CELLS * CELLS * 20
    device = _trace(product, s, key, bvh=P.BVH_LBVH)
    assert _worst(device[:-flux], one[:-flux]) < 1e-10


def test_mixed_batch(product):
    """An item whose tree has pairs in a batch with quadrics and dielectrics: the
    estimates are those of the item alone."""
    field = W.heliostat_field(product, n_helio=37, receiver_cells=7)[0]
    down = W.beam_down(product, n_helio=60, receiver_cells=5)[0]
    for launch in ("launch", "launch_noalloc"):
        b = P.Batch(product, [field, down])
        rng = field.rng(seed=3)
        getattr(b, launch)(rng, [30011, 20011])
        got = b.finish(rng)
        for s, e, n in ((field, got[0], 30011), (down, got[1], 20011)):
            alone, mixed = s.solve(n, seed=3).globals(), e.globals()
            for k in alone:
                assert mixed[k][0] == pytest.approx(alone[k][0], rel=1e-10, abs=1e-10), k
        b.close()
