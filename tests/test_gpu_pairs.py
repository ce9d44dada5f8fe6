"""Pairs of triangles change nothing but the node visits: where a ray meets two
triangles at one distance, on the edge they share, the tree decides which is
hit, and it must decide as with leaves of one. A receiver whose axes are the
scene's has some tens of such hits in 3e7 paths, and its flux map tells which
cell each went to. All sums, among them the map's, equal those of leaves of one
but for their order (1e-10: sums of positive FP64 terms)."""
import ctypes as C

import pytest
import torch

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu
PATHS = 30_000_000


def _scene(lib, normals):
    s = P.Scene(lib)
    sun, aim = W.to_sun(50.0, 180.0), (0.0, 0.0, 100.0)
    if normals:
        corners = [(-4, -4, 0), (4, -4, 0), (4, 4, 0), (-4, 4, 0)]
        shape = s.mesh(corners, [(0, 2, 1), (2, 0, 3)],
                       normals=[W._unit((0.001 * x, 0.001 * y, 1.0)) for x, y, _ in corners])
    else:
        shape = s.rectangle(4, 4)
    obj = s.object([(shape, s.mirror(0.9, 2e-3), s.matte(0.0))])
    for p in W.surround_layout(400):
        a = W._unit(tuple(aim[c] - p[c] for c in range(3)))
        s.instance(obj, P.transform_from(W.frame_z_to(W._unit(tuple(sun[c] + a[c] for c in range(3)))), p))
    m = s.mirror(0.05, 0.0)
    s.instance(s.object([(W.grid_mesh(s, 12.0, 12.0, 24, 24), m, m)]),
               P.transform_from(P.rotation_pitch_pi(), aim), receiver=P.SSOL_FRONT,
               per_primitive=1, sample=0)
    s.set_sun("pillbox", tuple(-x for x in sun), 900.0, param=4.65e-3)
    return s


def _sums(lib, s, leaf, seed):
    h = C.c_void_p()
    opt = P.options(leaf=leaf)
    lib.call("ssol_b200_plan_create", s.scn, C.byref(opt), C.byref(h))
    try:
        lib.call("ssol_b200_plan_launch", h, s.rng(seed=seed), 0, PATHS, None)
        torch.cuda.synchronize()
        return torch.as_tensor(P.plan_tallies(lib, h)[0], device="cuda").clone()
    finally:
        lib.raw("ssol_b200_plan_ref_put", h)


@pytest.mark.parametrize("normals", [False, True])
def test_hits_on_shared_edges(product, normals):
    s = _scene(product, normals)
    for seed in (5, 6, 7):
        a, b = _sums(product, s, 0, seed), _sums(product, s, 1, seed)
        worst = float(((a - b).abs() / b.abs().clamp(min=1e-300)).max())
        assert worst < 1e-10, (seed, worst)
