"""The sums that follow from others (a receiver side's, the global cosine and
shadowed) around the numbers of sampled instances at which one block no longer
adds them all up (2048) and at which its slices grow (65536), and of the slots
(400000) from which a block takes several receiver sides: they are the sums of
the per-instance ones, after each of two launches, in plans and batches. Both
are sums of the same positive FP64 numbers, so they differ by their order only
(n 2^-53 = 1e-11 at most; 1e-10)."""
import ctypes as C

import pytest
import torch

import pyssol as P

pytestmark = pytest.mark.gpu


def _scene(lib, n, k=0):
    """n mirrors of 1 m2 in a square grid under two receivers, front and back, or
    under k x k ones."""
    s = P.Scene(lib)
    m, rm = s.mirror(0.9, 1e-3), s.mirror(0.05, 0.0)
    o = s.object([(s.rectangle(0.5, 0.5), m, m)])
    side = int(n ** 0.5) + 1
    for i in range(n):
        s.instance(o, P.transform_from(None, (1.5 * (i % side), 1.5 * (i // side), 0.0)))
    w = 0.75 * side
    if k:
        rect = s.object([(s.rectangle(0.6 * w / k, 0.6 * w / k), rm, rm)])
    for i in range(k * k):
        s.instance(rect, P.transform_from(P.rotation_pitch_pi(),
                                          (w * (2 * (i % k) + 1) / k, w * (2 * (i // k) + 1) / k, 1.0)),
                   receiver=P.SSOL_FRONT | P.SSOL_BACK, sample=0)
    for x in () if k else (0.3 * w, 1.5 * w):
        s.instance(s.object([(s.rectangle(0.5 * w, w), rm, rm)]),
                   P.transform_from(P.rotation_pitch_pi(), (x, w, 30.0)),
                   receiver=P.SSOL_FRONT | P.SSOL_BACK, sample=0)
    s.set_sun("pillbox", (0.1, 0.3, -1.0), 1000.0, param=4.65e-3)
    return s


def _check(sums, n, nrcv=4):
    at, parts = 0, []
    for size in (12, nrcv * 20, n * 4, n * nrcv * 20):  # each from a multiple of 32
        parts.append(sums[at:at + size])
        at = (at + size + 31) // 32 * 32
    glob, rcv, samp, samp_rcv = parts
    want = samp_rcv.reshape(n, nrcv * 20).sum(0)
    assert float(want.max()) > 0
    torch.testing.assert_close(rcv, want, rtol=1e-10, atol=0)
    want = samp.reshape(n, 4).sum(0)
    torch.testing.assert_close(glob[[0, 1, 4, 5]], want, rtol=1e-10, atol=0)


@pytest.mark.parametrize("n,k", [(2047, 0), (2048, 0), (2049, 0), (4097, 0), (65537, 0),
                                 (887, 15), (889, 15), (95, 46), (97, 46), (22222, 3), (22223, 3),
                                 (99999, 0), (100000, 0)])
def test_sums_of_slices(product, n, k):
    s = _scene(product, n, k)
    h = C.c_void_p()
    opt = P.options()
    product.call("ssol_b200_plan_create", s.scn, C.byref(opt), C.byref(h))
    try:
        rng = s.rng(seed=4)
        for first in (0, 150001):
            product.call("ssol_b200_plan_launch", h, rng, first, 150001, None)
            torch.cuda.synchronize()
            sums, _ = P.plan_tallies(product, h)
            _check(torch.as_tensor(sums, device="cuda"), n, 2 * k * k or 4)
    finally:
        product.raw("ssol_b200_plan_ref_put", h)


def test_batch_of_small_and_large(product):
    """Slices are those of the largest item; the items alone give the same."""
    scenes = [_scene(product, n) for n in (3, 2500, 40)]
    for launch in ("launch", "launch_noalloc"):
        b = P.Batch(product, scenes)
        rng = scenes[0].rng(seed=9)
        for _ in range(2):
            getattr(b, launch)(rng, [20011, 40009, 0])
        for s, e, n in zip(scenes, b.finish(rng), (40022, 80018, 0)):
            if not n:
                continue
            alone = s.solve(n, seed=9).globals()
            got = e.globals()
            for k in alone:
                assert got[k][0] == pytest.approx(alone[k][0], rel=1e-10, abs=1e-10), k
        b.close()
