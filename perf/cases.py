"""Timing cases of the solver: the calls that its users make, over the sizes
and options they make them with, through the public C API (pyssol, the ctypes
binding, adds only the argument marshalling).

- `listed()`: named cases, from one small mirror to whole plants.
- `draw(rng)`: one more case of the same ranges.
- `prepare(case, seed)`: what a program holds before the call: the scene
  described through the API, and the plan or batch it keeps. The seed moves
  the sun, its DNI and the random streams.
- `run(state)`: one pass, returning the estimates, gradients or pixels.
- `work(case)`: bytes and operations no implementation can do without.
- `exact(case, seed)`: the same estimates in 64 bits by brute force (flat
  mirrors and heliostats under a pillbox or Gaussian sun, and the draft
  renderer), on the random streams that the C header documents.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "solstice-solver_b200"))
import adjoint as A  # noqa: E402
import pyssol as P  # noqa: E402
import workloads as W  # noqa: E402

_LIB = None
AIM = (0.0, 0.0, 100.0)
DRAW_CAMERA = ((0.0, -60.0, 170.0), (0.0, 280.0, 0.0), (0.0, 0.0, 1.0), math.radians(75.0))


def _lib():
    global _LIB
    if _LIB is None:
        _LIB = P.load_product()
    return _LIB


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A quick look at one mirror: the latency of a whole ssol_solve
        # (snapshot, tree, upload, launch, read-back).
        {"name": "mirror_solve_10k", "kind": "mirror", "paths": 10_000},
        # The single-mirror benchmark scene at its own size.
        {"name": "mirror_solve_1m", "kind": "mirror", "paths": 1_000_000},
        # A plant during its design: one ssol_solve per layout, coarse map.
        {"name": "field_solve_1m", "kind": "field", "helio": 1000, "cells": 24,
         "paths": 1_000_000, "sun": "pillbox", "fp64": False, "plan": False},
        # A mid-size plant under a sunshape with a circumsolar halo, an odd
        # number of realisations.
        {"name": "field_buie_solve_5m", "kind": "field", "helio": 317, "cells": 31,
         "paths": 5_123_457, "sun": "buie", "fp64": False, "plan": False},
        # The 1000-heliostat benchmark field resident on the device (plan),
        # 64 x 64 flux map, 1e8 realisations.
        {"name": "field_plan_100m", "kind": "field", "helio": 1000, "cells": 64,
         "paths": 100_000_000, "sun": "pillbox", "fp64": False, "plan": True},
        # The all-FP64 build, used to check the precision of a result.
        {"name": "field_fp64_solve_2m", "kind": "field", "helio": 500, "cells": 16,
         "paths": 2_000_003, "sun": "gaussian", "fp64": True, "plan": False},
        # Punched paraboloids, hyperboloid secondary, glass window: deep
        # paths through ssol_solve ...
        {"name": "beamdown_solve_4m", "kind": "beamdown", "helio": 1200, "cells": 20,
         "paths": 4_000_000, "plan": False},
        # ... and the 5000-heliostat benchmark scene as a plan.
        {"name": "beamdown_plan_60m", "kind": "beamdown", "helio": 5000, "cells": 30,
         "paths": 60_000_000, "plan": True},
        # Sun positions of a year as one batch, ragged budgets.
        {"name": "suns_batch_32", "kind": "suns", "helio": 1000, "cells": 8, "suns": 32,
         "lo": 100_000, "hi": 4_000_000},
        # Aim optimisation: objective and gradients (forward and backward).
        {"name": "adjoint_10m", "kind": "adjoint", "helio": 1000, "cells": 64,
         "paths": 10_000_000},
        # Preview images into device memory.
        {"name": "draft_1080p", "kind": "draft", "helio": 1000, "width": 1920,
         "height": 1080, "spp": 4},
        {"name": "pt_1080p", "kind": "pt", "helio": 1000, "width": 1920, "height": 1080,
         "spp": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mirror", "field", "field", "field", "field", "beamdown", "beamdown",
                       "suns", "adjoint", "draft", "pt"])
    if kind == "mirror":
        return {"kind": kind, "paths": _log(rng, 10_000, 10_000_000)}
    if kind == "field":
        fp64 = rng.random() < 0.2
        plan = rng.random() < 0.5
        top = 4_000_000 if fp64 else 100_000_000 if plan else 20_000_000
        return {"kind": kind, "helio": _log(rng, 30, 1000), "cells": rng.randint(4, 64 if plan else 32),
                "paths": _log(rng, 50_000, top), "sun": rng.choice(["pillbox", "gaussian", "buie"]),
                "fp64": fp64, "plan": plan}
    if kind == "beamdown":
        plan = rng.random() < 0.5
        return {"kind": kind, "helio": _log(rng, 100, 4000), "cells": rng.randint(6, 30),
                "paths": _log(rng, 100_000, 40_000_000 if plan else 10_000_000), "plan": plan}
    if kind == "suns":
        n = rng.randint(3, 48)
        return {"kind": kind, "helio": _log(rng, 50, 1000), "cells": rng.randint(4, 10),
                "suns": n, "lo": 20_000, "hi": _log(rng, 200_000, 4_000_000)}
    if kind == "adjoint":
        return {"kind": kind, "helio": _log(rng, 30, 1000), "cells": rng.randint(16, 80),
                "paths": _log(rng, 200_000, 20_000_000)}
    w = _log(rng, 320, 1920)
    return {"kind": kind, "helio": _log(rng, 50, 1000), "width": w,
            "height": max(120, int(w * rng.uniform(0.5, 0.75))),
            "spp": rng.randint(1, 8 if kind == "draft" else 16)}


# ----------------------------------------------------------------- prepare
def _inputs(seed):
    """What the seed decides: the sun, its DNI and the key of the streams."""
    r = random.Random(1000003 * seed + 17)
    return {"elevation": r.uniform(25.0, 60.0), "azimuth": r.uniform(150.0, 210.0),
            "dni": r.uniform(600.0, 1000.0), "key": r.randrange(1 << 40)}


def _field(case, inp):
    s, h = W.heliostat_field(_lib(), n_helio=case["helio"], elevation=inp["elevation"],
                             azimuth=inp["azimuth"], dni=inp["dni"],
                             receiver_cells=case.get("cells", 64))
    sun = case.get("sun", "pillbox")
    if sun != "pillbox":
        s.set_sun(sun, tuple(-c for c in h["sun"]), inp["dni"],
                  param=2.5e-3 if sun == "gaussian" else 0.05)
    return s, h


class _Plan:
    """A resident plan and its stream keys, released with the state."""

    def __init__(self, scene, key):
        self.scene = scene
        self.h = C.c_void_p()
        scene.lib.call("ssol_b200_plan_create", scene.scn, None, C.byref(self.h))
        self.rng = scene.rng(seed=key)

    def __del__(self):
        if self.h:
            self.scene.lib.raw("ssol_b200_plan_ref_put", self.h)
            self.h = None


def prepare(case, seed):
    kind, inp = case["kind"], _inputs(seed)
    st = {"kind": kind, "case": case}
    if kind == "mirror":
        s, h = W.single_mirror(_lib())
        s.set_sun("pillbox", _mirror_sun(inp), inp["dni"], param=4.65e-3)
        st.update(scene=s, h=h, rng=s.rng(seed=inp["key"]), cells=0, opts=None, plan=None)
    elif kind in ("field", "beamdown"):
        if kind == "field":
            s, h = _field(case, inp)
        else:
            s, h = W.beam_down(_lib(), n_helio=case["helio"], elevation=inp["elevation"] + 15.0,
                               azimuth=inp["azimuth"], dni=inp["dni"],
                               receiver_cells=case["cells"])
        st.update(scene=s, h=h, cells=case["cells"], rng=s.rng(seed=inp["key"]),
                  opts=P.options(precision=P.FP64) if case.get("fp64") else None,
                  plan=_Plan(s, inp["key"]) if case["plan"] and not case.get("fp64") else None)
    elif kind == "suns":
        s, h = _field(case, inp)
        r = random.Random(seed + 5)
        suns = [{"elevation": r.uniform(10.0, 80.0), "azimuth": r.uniform(90.0, 270.0),
                 "dni": r.uniform(300.0, 1000.0)} for _ in range(case["suns"])]
        # the same budgets for every seed, so that every state is the same work
        b = random.Random(case["suns"])
        st["budgets"] = [_log(b, case["lo"], case["hi"]) for _ in suns]
        st.update(scene=s, h=h, rng=s.rng(seed=inp["key"]),
                  batch=P.Batch.tracking(s, *W.tracking_inputs(h, suns, AIM)))
    elif kind == "adjoint":
        s, h = _field(case, inp)
        r = random.Random(seed + 9)
        field = A.AimField(s, h["heliostats"], h["transforms"], h["receiver"], (-6.0, -6.0),
                           (6.0, 6.0), case["cells"], case["cells"],
                           100.0 * case["helio"] * inp["dni"] * 0.5 / 144.0, case["paths"],
                           seed=inp["key"])
        field.apply([(r.uniform(-2e-3, 2e-3), r.uniform(-2e-3, 2e-3)) for _ in h["heliostats"]])
        st["field"] = field
    else:
        s, h = _field(dict(case, cells=64), inp)
        ground = s.matte(0.3)
        s.instance(s.object([(s.rectangle(2000, 2000), ground, ground)]),
                   P.transform_from(None, (0.0, 0.0, -0.5)), sample=0)
        pos, tgt, up, fov = DRAW_CAMERA
        st.update(scene=s, cam=s.camera(pos, tgt, up, fov=fov, ratio=case["width"] / case["height"]),
                  seed=inp["key"], pixels=torch.empty((case["height"], case["width"], 3),
                                                      dtype=torch.float64, device="cuda"))
    return st


def _mirror_sun(inp):
    """From the sun toward the mirror, within 20 mrad of the 45 degrees that
    send its reflection to the receiver's centre."""
    c = math.cos(math.pi / 4)
    a = (inp["elevation"] - 42.5) * 1e-3
    b = (inp["azimuth"] - 180.0) * 1e-3 / 2
    v = (b, c + a * c, -c + a * c)
    n = math.sqrt(sum(x * x for x in v))
    return tuple(x / n for x in v)


# --------------------------------------------------------------------- run
def _ev(structs):
    """E and V of an array of (E, V, SE) results (SE is sqrt(V / N))."""
    a = np.frombuffer(structs, dtype=np.float64).reshape(-1, 3)
    return {"E": a[:, 0].copy(), "V": a[:, 1].copy()}


def _results(lib, est, h, cells):
    """The global estimates, the receiver's, and its flux map."""
    g, r = P.McGlobal(), P.McReceiver()
    lib.call("ssol_estimator_get_mc_global", est, C.byref(g))
    lib.call("ssol_estimator_get_mc_receiver", est, h["receiver"], P.SSOL_FRONT, C.byref(r))
    out = {"global": _ev(g),
           "receiver": _ev((P.McResult * len(P.RCV_FIELDS)).from_buffer(r))}
    if cells:
        n, size = 2 * cells * cells, C.sizeof(P.McPrimitive)
        ms, prims = P.McShape(), (P.McPrimitive * n)()
        lib.call("ssol_mc_receiver_get_mc_shape", C.byref(r), h["receiver_shape"], C.byref(ms))
        get = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_uint, C.c_void_p)(
            ("ssol_mc_shape_get_mc_primitive", lib.dll))
        at, base = C.addressof(ms), C.addressof(prims)
        for i in range(n):
            get(at, i, base + i * size)
        out["map"] = _ev(prims)
    return out


def run(st):
    kind, case = st["kind"], st["case"]
    if kind in ("mirror", "field", "beamdown"):
        s, est = st["scene"], C.c_void_p()
        plan = st["plan"]
        if plan is None:
            if st["opts"] is None:
                res = s.lib.raw("ssol_solve", s.scn, st["rng"], case["paths"], 1 << 40, None,
                                C.byref(est))
            else:
                res = s.lib.raw("ssol_solve_ex", s.scn, st["rng"], case["paths"], 1 << 40, None,
                                C.byref(st["opts"]), C.byref(est))
            if res != P.RES_OK:
                raise P.SsolError("ssol_solve", res)
            out = _results(s.lib, est, st["h"], st["cells"])
        else:
            s.lib.call("ssol_b200_plan_reset", plan.h, None)
            s.lib.call("ssol_b200_plan_launch", plan.h, plan.rng, 0, case["paths"], None)
            s.lib.call("ssol_b200_plan_finish", plan.h, plan.rng, case["paths"], 1 << 40, None,
                       C.byref(est))
            out = _results(s.lib, est, st["h"], 0)
            # The sums behind every estimate (flux map and per-heliostat
            # results included), a copy on the device: the plan's own
            # buffer ends with the plan
            sums, counts = P.plan_tallies(s.lib, plan.h)
            out["sums"] = torch.as_tensor(sums, device="cuda").clone()
            out["samples"] = torch.as_tensor(counts, device="cuda")[:case["helio"]].clone()
        s.lib.raw("ssol_estimator_ref_put", est)
        return out
    if kind == "suns":
        b, lib = st["batch"], st["scene"].lib
        b.reset()
        b.launch(st["rng"], st["budgets"])
        items = [_results(lib, e.h, st["h"], case["cells"])
                 for e in b.finish(st["rng"], max_failed=1 << 40)]
        return {k: {q: np.stack([r[k][q] for r in items]) for q in ("E", "V")}
                for k in ("global", "receiver", "map")}
    if kind == "adjoint":
        r = st["field"].evaluate(gradients=True, want_map=True)
        return {"absorbed": r["absorbed"], "spillage": r["spillage"], "hits": int(r["hits"]),
                "d_absorbed": np.array(r["d_absorbed"]),
                "d_spillage": np.array(r["d_spillage"]), "map": np.array(r["map"])}
    st["scene"].draw_device(kind, st["cam"], case["width"], case["height"], case["spp"],
                            st["pixels"].data_ptr(), seed=st["seed"])
    return st["pixels"]


# -------------------------------------------------------------------- work
def work(case):
    """Operations of a path: one primary sample (120), per ray the two box
    tests of every level of a balanced tree (40 each) and one primitive test
    (55 a triangle, 90 a quadric), per reflection 150. Bytes: the scene's
    primitives in, the sums or pixels out."""
    kind = case["kind"]
    if kind == "mirror":
        return {"bytes": 4 * 48 + 8 * 60, "flops": case["paths"] * (120 + 2 * (40 + 55) + 150)}
    helio = case["helio"]
    tris = 2 * helio + 2 * case.get("cells", 64) ** 2
    levels = math.ceil(math.log2(tris))
    if kind == "beamdown":
        prims = helio + 3 + 2 * case["cells"] ** 2
        ray = 40 * math.ceil(math.log2(prims)) + 90
        return {"bytes": 100 * prims + 160 * (2 * case["cells"] ** 2 + helio),
                "flops": case["paths"] * (120 + 4 * ray + 3 * 150)}
    ray = 40 * levels + 55
    if kind == "field":
        k = 2 if case["fp64"] else 1
        return {"bytes": 48 * k * tris + 160 * (2 * case["cells"] ** 2 + helio),
                "flops": case["paths"] * (120 + 2 * ray + 150)}
    if kind == "suns":
        b = random.Random(case["suns"])
        paths = sum(_log(b, case["lo"], case["hi"]) for _ in range(case["suns"]))
        return {"bytes": case["suns"] * (48 * tris + 160 * (2 * case["cells"] ** 2 + helio)),
                "flops": paths * (120 + 2 * ray + 150)}
    if kind == "adjoint":
        return {"bytes": 48 * tris + 8 * case["cells"] ** 2 + 32 * helio,
                "flops": case["paths"] * 2 * (120 + 2 * ray + 150)}
    px = case["width"] * case["height"]
    rays = px * case["spp"] * (2 if kind == "pt" else 1)
    return {"bytes": 48 * tris + 24 * px, "flops": rays * ray}


# ------------------------------------------------------------------- exact
# Brute force in 64 bits over rectangles: rows of centre, x, y, n (unit
# vectors), half sizes.
def _rect(R, c, half):
    return [*c, R[0][0], R[1][0], R[2][0], R[0][1], R[1][1], R[2][1], R[0][2], R[1][2], R[2][2],
            half]


def _philox(ids, event, domain, key):
    """Philox4x32-10 block (id, event, domain) of every id: four uniforms of
    24 bits."""
    m = 0xFFFFFFFF
    c = [ids & m, ids >> 32, torch.full_like(ids, event), torch.full_like(ids, domain)]
    k0, k1 = key & m, key >> 32 & m

    def mul(a, x):  # 32 x 32 bits -> high and low words, in two halves
        lo, hi = a * (x & 0xFFFF), a * (x >> 16)
        t = (lo >> 16) + (hi & 0xFFFF)
        return (hi >> 16) + (t >> 16), (t & 0xFFFF) << 16 | lo & 0xFFFF

    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    return [(x >> 8).double() * 2.0 ** -24 for x in c]


def _basis(n):
    s = torch.where(n[:, 2] >= 0, 1.0, -1.0).double()
    a = -1.0 / (s + n[:, 2])
    b = n[:, 0] * n[:, 1] * a
    return (torch.stack([1 + s * n[:, 0] ** 2 * a, s * b, -s * n[:, 0]], 1),
            torch.stack([b, s + n[:, 1] ** 2 * a, -n[:, 1]], 1))


def _cast(rects, org, d, skip):
    """First rectangle along each ray (-1: none) and its distance; `skip` is
    the one the ray leaves."""
    best_t, best = [], []
    c, x, y, n, half = (rects[:, 0:3], rects[:, 3:6], rects[:, 6:9], rects[:, 9:12], rects[:, 12])
    step = max(1, 40_000_000 // len(rects))
    for i in range(0, max(1, len(org)), step):
        o, v = org[i:i + step], d[i:i + step]
        t = ((c * n).sum(1) - o @ n.T) / (v @ n.T)
        u = (o @ x.T - (c * x).sum(1)) + t * (v @ x.T)
        w = (o @ y.T - (c * y).sum(1)) + t * (v @ y.T)
        bad = ~((u.abs() <= half) & (w.abs() <= half) & (t > 1e-9))
        bad |= torch.arange(len(rects), device=t.device) == skip[i:i + step, None]
        t = t.masked_fill(bad, math.inf)
        m = t.min(1)
        best_t.append(m.values)
        best.append(torch.where(m.values < math.inf, m.indices, -1))
    return torch.cat(best), torch.cat(best_t)


def _moments(per_path, n):
    """E and V of the columns of per-path totals."""
    e = per_path.sum(0) / n
    v = ((per_path ** 2).sum(0) / n - e ** 2).clamp(min=0)
    return {"E": e.cpu().numpy(), "V": v.cpu().numpy()}


def _solve64(rects, mirrors, back_black, refl, slope, cells, sun, kind, param, dni, kext, n, key):
    """The realisation loop on rectangles: `mirrors` sampled ones, then the
    receiver (front side, reflectivity 0.05)."""
    dev = "cuda"
    rects = torch.tensor(rects, dtype=torch.float64, device=dev)
    rcv = len(rects) - 1
    mats = torch.tensor([[refl, slope], [0.05, 0.0]], dtype=torch.float64, device=dev)
    ids = torch.arange(n, dtype=torch.int64, device=dev)
    r0, r1 = _philox(ids, 0, 0, key), _philox(ids, 1, 0, key)
    tri = (r0[0] * (2 * mirrors)).long()
    at, tri = tri // 2, tri % 2
    sa = r0[2].sqrt()
    b2 = sa * r0[3]
    b1 = sa - b2
    hf = rects[at, 12]
    # the rectangle's triangles: corners (0, 2, 1) and (2, 0, 3)
    px = torch.where(tri == 0, -hf + 2 * hf * b1 + 2 * hf * b2, hf - 2 * hf * b1 - 2 * hf * b2)
    py = torch.where(tri == 0, -hf + 2 * hf * b1, hf - 2 * hf * b1)
    pos = rects[at, 0:3] + px[:, None] * rects[at, 3:6] + py[:, None] * rects[at, 6:9]
    s0 = torch.tensor(sun, dtype=torch.float64, device=dev)
    s0 = s0 / s0.norm()
    if kind == "pillbox":
        st = (r1[0] * math.sin(param) ** 2).sqrt()
    else:
        st = (param * (-2 * torch.log(1 - r1[0])).sqrt()).clamp(max=1.0)
    phi = 2 * math.pi * r1[1]
    e1, e2 = _basis(s0[None])
    d = (st * phi.cos())[:, None] * e1 + (st * phi.sin())[:, None] * e2 + (1 - st ** 2).sqrt()[:, None] * s0
    nrm = rects[at, 9:12]
    back = (nrm * d).sum(1) >= 0
    N = torch.where(back[:, None], -nrm, nrm)
    area = 4 * (rects[:mirrors, 12] ** 2).sum()
    w0 = dni * area * ((N * d).sum(1) / (d @ s0)).abs()
    g = torch.zeros(n, 6, dtype=torch.float64, device=dev)
    g[:, 0] = (N @ s0).abs()
    hit, _ = _cast(rects, pos, -d, at)
    g[:, 2] = torch.where(hit >= 0, w0, 0.0)
    live = torch.nonzero(hit < 0)[:, 0]
    rp = torch.zeros(n, 6, dtype=torch.float64, device=dev)
    cell_key, cell_val = [], []
    on, pos, d, N, back = at[live], pos[live], d[live], N[live], back[live]
    w = torch.stack([w0[live]] * 3, 1)
    dist = torch.zeros(len(live), dtype=torch.float64, device=dev)
    for event in range(60):
        if not len(live):
            break
        inc = w.clone()
        tr = torch.exp(-kext * dist)
        inc[:, 0] *= tr
        inc[:, 2] *= tr
        g[live, 4] += w[:, 0] - inc[:, 0]
        wo = -d
        ci = (wo * N).sum(1)
        is_rcv = on == rcv
        r = _philox(ids[live], event, 1, key)
        rough = torch.where(is_rcv, mats[1, 1], mats[0, 1])
        tan2 = -rough ** 2 * torch.log(1 - r[0])
        ct = 1 / (1 + tan2).sqrt()
        sn = tan2.sqrt() * ct
        f1, f2 = _basis(N)
        hm = (sn * (2 * math.pi * r[1]).cos())[:, None] * f1 + (sn * (2 * math.pi * r[1]).sin())[:, None] * f2 + ct[:, None] * N
        wh = (wo * hm).sum(1)
        out = 2 * wh[:, None] * hm - wo
        pr = torch.where(is_rcv, mats[1, 0], mats[0, 0])
        if back_black:
            pr = torch.where(back & ~is_rcv, 0.0, pr)
        pr = torch.where((ci > 0) & (wh > 0) & ((out * N).sum(1) > 0), pr, 0.0)
        took = is_rcv & ~back
        val = torch.cat([inc, inc * (1 - pr)[:, None]], 1)
        rp.index_add_(0, live[took], val[took])
        g[live, 1] += torch.where(took, inc[:, 0] * (1 - pr), 0.0)
        g[live, 5] += torch.where(took, 0.0, inc[:, 0] * (1 - pr))
        if cells and bool(took.any()):
            q = pos[took] - rects[rcv, 0:3]
            hfr = float(rects[rcv, 12])
            u = (q @ rects[rcv, 3:6] + hfr) / (2 * hfr) * cells
            v = (q @ rects[rcv, 6:9] + hfr) / (2 * hfr) * cells
            iu, iv = u.long().clamp(0, cells - 1), v.long().clamp(0, cells - 1)
            # quad (a, c, b), (c, a, d): first triangle below the diagonal
            prim = 2 * (iv * cells + iu) + ((v - iv) > (u - iu)).long()
            cell_key.append(live[took] * (2 * cells * cells) + prim)
            cell_val.append(val[took])
        w = inc * pr[:, None]
        w[:, 2] = torch.where(took, w[:, 2], inc[:, 2])
        keep = pr > 0
        live, pos, d, w, on = live[keep], pos[keep], out[keep], w[keep], on[keep]
        hit, dist = _cast(rects, pos, d, on)
        gone = hit < 0
        g[live[gone], 3] += w[gone, 0]
        live, pos, d, w, on, dist = (x[~gone] for x in (live, pos, d, w, hit, dist))
        pos = pos + dist[:, None] * d
        nrm = rects[on, 9:12]
        back = (nrm * d).sum(1) >= 0
        N = torch.where(back[:, None], -nrm, nrm)

    def ten(v):
        a, b = v[:, :3], v[:, 3:]
        return torch.cat([a, a[:, 2:3] - a[:, :1], a[:, 1:2] - a[:, :1],
                          b, b[:, 2:3] - b[:, :1], b[:, 1:2] - b[:, :1]], 1)

    res = {"global": _moments(g, n), "receiver": _moments(ten(rp), n)}
    if cells:
        np_ = 2 * cells * cells
        key_, inv = torch.unique(torch.cat(cell_key), return_inverse=True)
        v = torch.zeros(len(key_), 6, dtype=torch.float64, device=dev)
        v = ten(v.index_add_(0, inv, torch.cat(cell_val)))
        a = (2 * float(rects[rcv, 12])) ** 2 / np_
        s1 = torch.zeros(np_, 10, dtype=torch.float64, device=dev).index_add_(0, key_ % np_, v / a)
        s2 = torch.zeros(np_, 10, dtype=torch.float64, device=dev).index_add_(0, key_ % np_, (v / a) ** 2)
        e = s1 / n
        res["map"] = {"E": e.reshape(-1).cpu().numpy(),
                      "V": (s2 / n - e ** 2).clamp(min=0).reshape(-1).cpu().numpy()}
    return res


def _field_rects(helio, sun, with_ground):
    pts = W.field_layout(helio)
    rects = []
    for p in pts:
        a = W._unit(tuple(AIM[c] - p[c] for c in range(3)))
        nn = W._unit(tuple(sun[c] + a[c] for c in range(3)))
        rects.append(_rect(W.frame_z_to(nn), p, 5.0))
    if with_ground:
        rects.append(_rect(((1, 0, 0), (0, 1, 0), (0, 0, 1)), (0.0, 0.0, -0.5), 2000.0))
    ctr = [sum(p[c] for p in pts) / len(pts) for c in range(3)]
    rects.append(_rect(W.frame_z_to(W._unit(tuple(ctr[c] - AIM[c] for c in range(3)))), AIM, 6.0))
    return rects


def exact(case, seed):
    kind, inp = case["kind"], _inputs(seed)
    if kind == "mirror" and case["paths"] <= 4_000_000:
        c = math.cos(math.pi / 4)
        rc = (0.0, c, c)
        R = W.frame_z_to(tuple(-x for x in rc), up=(1.0, 0.0, 0.0))
        rects = [_rect(((1, 0, 0), (0, 1, 0), (0, 0, 1)), (0.0, 0.0, 0.0), 5.0),
                 _rect(R, tuple(50 * x for x in rc), 2.0)]
        return _solve64(rects, 1, False, 0.9, 0.0, 0, _mirror_sun(inp), "pillbox", 4.65e-3,
                        inp["dni"], 0.0, case["paths"], inp["key"])
    sun = W.to_sun(inp["elevation"], inp["azimuth"])
    if kind == "field" and not case["plan"] and case["sun"] != "buie" and case["paths"] <= 2_500_000:
        # (Buie: its rejection loop; larger ones: the time)
        return _solve64(_field_rects(case["helio"], sun, False), case["helio"], True, 0.9, 2e-3,
                        case["cells"], tuple(-x for x in sun), case["sun"],
                        4.65e-3 if case["sun"] == "pillbox" else 2.5e-3, inp["dni"], 1e-4,
                        case["paths"], inp["key"])
    if kind == "draft":
        return _draft64(case, sun)
    # Beam-down, batches, adjoints and path tracing: brute force over their
    # paths takes minutes
    return None


def _draft64(case, sun):
    """The draft's pixels: mean over the sub-pixel offsets of the cosine
    between the first surface's normal and the ray."""
    dev, f8 = "cuda", torch.float64
    rects = torch.tensor(_field_rects(case["helio"], sun, True), dtype=f8, device=dev)
    pos, tgt, up, fov = (torch.tensor(v, dtype=f8) for v in DRAW_CAMERA)
    z = (tgt - pos) / (tgt - pos).norm()
    x = torch.linalg.cross(z, up)
    x = x / x.norm()
    y = torch.linalg.cross(z, x)
    y = y / y.norm() / (case["width"] / case["height"])
    z = z / math.tan(float(fov) / 2)
    x, y, z, pos = (v.to(dev) for v in (x, y, z, pos))
    wid, hei = case["width"], case["height"]
    img = torch.zeros(hei * wid, dtype=f8, device=dev)
    r = _philox(torch.arange(case["spp"], dtype=torch.int64), 0, 4, 0)
    jj, ii = torch.meshgrid(torch.arange(hei, device=dev), torch.arange(wid, device=dev), indexing="ij")
    none = torch.full((hei * wid,), -1, device=dev)
    for k in range(case["spp"]):
        fx = (ii.reshape(-1) + float(r[0][k])) / wid * 2 - 1
        fy = (jj.reshape(-1) + float(r[1][k])) / hei * 2 - 1
        d = fx[:, None] * x + fy[:, None] * y + z
        d = d / d.norm(dim=1, keepdim=True)
        hit, _ = _cast(rects, pos.expand_as(d), d, none)
        c = (rects[hit.clamp(min=0), 9:12] * d).sum(1).abs()
        img += torch.where(hit >= 0, c, 0.0)
    img = (img / case["spp"]).reshape(hei, wid, 1)
    return img.expand(hei, wid, 3).contiguous()
