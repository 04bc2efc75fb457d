"""Performance cases: what a program built on this library has it do.

Each case goes through the public Python objects (experiments_b200.b3): a world
that steps from a written state, the adjoint of a rollout, and the sort, search
and scan primitives. A stepping program keeps its world (shapes, bodies, device
buffers, launch shapes) and writes a new state into the borrowed device views
before it steps, as a simulator that resets its environments does; the state is
written again on every pass, so every pass does the same work.

Scenes are made here from the seed alone. `packing` says how the bodies lie:
"falling" is a lattice in the air with gaps, few pairs touching, as a scene
begins; "settled" is a heap, bodies turned every way and a few millimetres to a
few centimetres inside their neighbours, as it looks for most of a run.
"""
import functools
import math

import numpy as np
import torch

from experiments_b200 import b3, scenes

KINDS = ("step", "step", "step", "step", "step", "step", "adjoint", "sort", "cells")


def listed():
    return [
        # one small scene stepped interactively: latency of the captured step
        dict(name="cubes_4k", kind="step", shapes="cubes", bodies=4096, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=False),
        # the benchmark's mixed scene in a heap, launch shapes tuned once
        dict(name="mixed_131k_settled", kind="step", shapes="mixed", bodies=131072, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=True),
        # the large scene: a million stacked cubes
        dict(name="cubes_1m", kind="step", shapes="cubes", bodies=1048576, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=False),
        # thousands of uneven worlds in one step (8 to 512 bodies each)
        dict(name="piles_4096_worlds", kind="step", shapes="hulls", bodies=118, worlds=4096, packing="settled",
             broadphase="grid", solver="jacobi", autotune=True),
        # the reference demo's default broadphase, while the scene still falls
        dict(name="mixed_33k_sap", kind="step", shapes="mixed", bodies=33001, worlds=1, packing="falling",
             broadphase="sap", solver="jacobi", autotune=False),
        # the reference's GPU solver
        dict(name="mixed_65k_gs", kind="step", shapes="mixed", bodies=65537, worlds=1, packing="settled",
             broadphase="grid", solver="gs", autotune=False),
        # granular spheres on a plane
        dict(name="spheres_20k", kind="step", shapes="spheres", bodies=20011, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=False),
        # compounds of cubes with hulls among them
        dict(name="compounds_6k", kind="step", shapes="compounds", bodies=6000, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=False),
        # bodies on a triangle-mesh terrain
        dict(name="terrain_2k", kind="step", shapes="terrain", bodies=2048, worlds=1, packing="settled",
             broadphase="grid", solver="jacobi", autotune=False),
        # gradients of a throw with respect to velocities, masses and friction
        dict(name="throw_256_worlds", kind="adjoint", bodies=64, worlds=256, steps=16, every=8),
        # the reference's sort benchmark size, as (key, value) pairs
        dict(name="sort_4m", kind="sort", n=4194304, form="kv", bits=32),
        # cell lists from (cell, body) records: sort, count per cell, offsets
        dict(name="cells_100k", kind="cells", n=100003, cells=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(KINDS)
    if kind == "step":
        shapes = rng.choice(["cubes", "cubes", "mixed", "mixed", "hulls", "spheres", "compounds", "terrain"])
        worlds = 1
        if shapes in ("hulls",) or (shapes in ("cubes", "mixed") and rng.random() < 0.25):
            worlds = _log_int(rng, 16, 4096)
        if worlds > 1:
            bodies = _log_int(rng, 16, min(512, 480000 // worlds))
        else:
            bodies = _log_int(rng, *{"cubes": (512, 600000), "mixed": (512, 200000), "spheres": (1000, 60000),
                                     "compounds": (500, 12000), "terrain": (256, 6000)}[shapes])
        special = shapes in ("spheres", "compounds", "terrain")
        broadphase = "sap" if worlds == 1 and not special and bodies <= 70000 and rng.random() < 0.25 else "grid"
        solver = "gs" if not special and rng.random() < 0.2 else "jacobi"
        packing = "settled" if special else rng.choice(["settled", "settled", "falling"])
        return dict(kind=kind, shapes=shapes, bodies=bodies, worlds=worlds, packing=packing, broadphase=broadphase,
                    solver=solver, autotune=False)
    if kind == "adjoint":
        return dict(kind=kind, bodies=_log_int(rng, 8, 125), worlds=_log_int(rng, 16, 256), steps=rng.randint(4, 16),
                    every=rng.choice([4, 8]))
    if kind == "sort":
        return dict(kind=kind, n=_log_int(rng, 1000, 16000000), form=rng.choice(["kv", "keys", "records"]),
                    bits=rng.choice([32, 32, 24, 20, 16]))
    return dict(kind=kind, n=_log_int(rng, 1000, 8000000), cells=_log_int(rng, 512, 2000000))


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
# lattice spacing per packing and shape set: (horizontal, vertical)
SPACING = {
    ("settled", "cubes"): (1.22, 0.995),
    ("settled", "mixed"): (0.98, 0.94),
    ("settled", "hulls"): (0.98, 0.94),
    ("settled", "spheres"): (0.74, 0.70),
    ("settled", "compounds"): (2.1, 1.0),
    ("settled", "terrain"): (1.0, 0.95),
}
FALLING = 1.2


def _lattice(n, footprint):
    """n lattice cells (x, y, z), bottom layers first, at most `footprint`
    cells along x and z; ordered by x, y, z like the scenes module's."""
    i = np.arange(n)
    cells = np.stack([(i // footprint) % footprint, i // (footprint * footprint), i % footprint], 1)
    return cells[np.lexsort((cells[:, 2], cells[:, 1], cells[:, 0]))].astype(np.float64)


def _pow2(x):
    return max(4, 1 << int(math.ceil(math.log2(max(x, 1.0)))))


def _counts(case):
    """Bodies per world: uneven around the mean, as piles of one batch are (the
    case's own numbers, the same for every seed)."""
    w = case["worlds"]
    if w == 1:
        return np.array([case["bodies"]])
    mean = case["bodies"]
    # log-uniform over the range whose mean is the case's (8 to 512 at 118)
    c = np.exp(scenes.uniform(w, 10, w, math.log(8), math.log(513)))
    return np.clip(np.floor(c * mean / 118.0), 4, 640).astype(np.int64)


def _scene(case, seed):
    shapes_of, packing, worlds = case["shapes"], case["packing"], case["worlds"]
    counts = _counts(case)
    total = int(counts.sum())
    wid = np.repeat(np.arange(worlds), counts)
    if packing == "falling":
        sx = sy = FALLING
        jitter = 0.02
    else:
        sx, sy = SPACING[(packing, shapes_of)]
        jitter = 0.002 if shapes_of == "cubes" else 0.03
    if worlds > 1:
        cells = np.concatenate([_lattice(int(c), 4) for c in counts])
        foot = 4
    else:
        # a footprint twice as wide as it is high
        foot = max(4, int(round((2.0 * total) ** (1.0 / 3.0))))
        cells = _lattice(total, foot)
    y0 = 0.5 * sy if packing == "settled" else 1.0
    pos = (cells - [(foot - 1) / 2.0, 0.0, (foot - 1) / 2.0]) * [sx, sy, sx] + [0.0, y0, 0.0]
    pos += scenes.uniform(seed, 1, 3 * total, -jitter, jitter).reshape(total, 3)
    if shapes_of == "cubes" or packing == "falling":
        quat = scenes.yaw_quat(scenes.uniform(seed, 2, total, 0.0, 2 * np.pi))
        if packing == "settled":  # stacked cubes rest tilted by a few milliradians
            quat[:, [0, 2]] += scenes.normal(seed, 12, 2 * total, 0.002).reshape(total, 2)
            quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    elif shapes_of == "spheres":
        quat = np.tile([0.0, 0.0, 0.0, 1.0], (total, 1))
    else:
        quat = scenes.normal(seed, 2, 4 * total).reshape(total, 4)
        quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    mass = scenes.uniform(seed, 3, total, 0.5, 2.0)
    fric = scenes.uniform(seed, 4, total, 0.3, 0.9)
    pick = scenes.uniform(seed, 5, total)
    which = scenes.uniform(seed, 6, total)
    half = 100.0 if worlds == 1 else 10.0
    ground = scenes.box_vertices(half, 0.5, half)
    cube = scenes.box_vertices(0.5, 0.5, 0.5)
    pool = 64
    cell = 1.2 if packing == "falling" else 1.0
    ground_pos = [0.0, -0.5, 0.0]
    if shapes_of == "cubes":
        shapes, sid = [ground, cube], np.ones(total, np.int32)
    elif shapes_of == "mixed":  # half cubes, a quarter hulls, a quarter icospheres
        shapes = [ground, cube, scenes.icosphere_vertices(0.5)] + scenes.hull_pool(seed, pool)
        sid = np.where(pick < 0.5, 1, np.where(pick < 0.75, 2, 3 + (which * pool).astype(np.int32) % pool))
    elif shapes_of == "hulls":  # cubes and 12-point hulls
        shapes = [ground, cube] + scenes.hull_pool(seed, pool)
        sid = np.where(pick < 0.5, 1, 2 + (which * pool).astype(np.int32) % pool)
    elif shapes_of == "spheres":
        shapes = [{"kind": "plane", "normal": [0.0, 1.0, 0.0], "constant": 0.0}]
        shapes += [{"kind": "sphere", "radius": r} for r in _radii(seed)]
        sid = 1 + (which * len(_radii(seed))).astype(np.int32) % len(_radii(seed))
        ground_pos = [0.0, 0.0, 0.0]
        pos[:, 1] += 0.1
    elif shapes_of == "compounds":
        q90 = [0.0, math.sin(math.pi / 4), 0.0, math.cos(math.pi / 4)]
        one = [0.0, 0.0, 0.0, 1.0]
        shapes = [ground, cube] + scenes.hull_pool(seed, 4)
        shapes.append({"kind": "compound", "children": [(1, (0.55, 0.0, 0.0), one), (1, (-0.55, 0.0, 0.0), one)]})
        shapes.append({"kind": "compound", "children": [(1, (0.0, 0.0, 0.0), one), (1, (1.05, 0.0, 0.0), q90),
                                                        (1, (0.0, 0.0, 1.05), q90)]})
        sid = np.where(pick < 0.35, 6, np.where(pick < 0.7, 7, 2 + (which * 4).astype(np.int32) % 4))
        quat = scenes.yaw_quat(scenes.uniform(seed, 2, total, 0.0, 2 * np.pi))
        cell = 2.0
        pos[:, 1] += 0.1
    else:  # terrain
        size = 1.25 * foot * sx
        side = max(8, int(size))
        g = side + 1
        hx = (np.arange(g) / side - 0.5) * size
        X, Z = np.meshgrid(hx, hx, indexing="ij")
        Y = scenes.uniform(seed, 7, g * g, 0.0, 0.3).reshape(g, g)
        verts = np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1).astype(np.float32)
        a = (np.arange(side)[:, None] * g + np.arange(side)[None, :]).ravel()
        idx = np.stack([a, a + 1, a + g, a + g, a + 1, a + g + 1], 1).ravel().astype(np.int32)
        shapes = [{"kind": "mesh", "vertices": verts, "indices": idx}, cube] + scenes.hull_pool(seed, 4)
        sid = np.where(pick < 0.5, 1, 2 + (which * 4).astype(np.int32) % 4)
        ground_pos = [0.0, 0.0, 0.0]
        pos[:, 1] += 0.25
    speed = 0.2 if packing == "settled" else 0.5
    g = _grounds(worlds, ground_pos)
    f32 = np.float32
    return scenes.Scene(
        name="perf", shapes=shapes, num_worlds=worlds,
        shape=np.concatenate([np.zeros(worlds, np.int32), sid]).astype(np.int32),
        mass=np.concatenate([np.zeros(worlds), mass]).astype(f32),
        pos=np.concatenate([g, pos]).astype(f32),
        quat=np.concatenate([np.tile([0.0, 0.0, 0.0, 1.0], (worlds, 1)), quat]).astype(f32),
        friction=np.concatenate([np.full(worlds, 0.6), fric]).astype(f32),
        world=np.concatenate([np.arange(worlds), wid]).astype(np.int32),
        lin=np.concatenate([np.zeros((worlds, 3)), scenes.normal(seed, 8, 3 * total, speed).reshape(total, 3)]).astype(f32),
        ang=np.concatenate([np.zeros((worlds, 3)), scenes.normal(seed, 9, 3 * total, speed).reshape(total, 3)]).astype(f32),
        config=_config(cell, foot * sx, (cells[:, 1].max() + 1) * sy + 2.0, worlds, total))


@functools.lru_cache(maxsize=4)
def _radii(seed):
    return tuple(float(np.float32(r)) for r in scenes.uniform(seed, 11, 32, 0.3, 0.4))


def _grounds(worlds, at):
    return np.tile(np.asarray(at, np.float64), (worlds, 1))


def _config(cell, width, height, worlds, total):
    if worlds > 1:
        dims = (16, 16, 16)
    else:
        dims = (min(256, _pow2(1.2 * width / cell)), min(256, _pow2(1.2 * height / cell)),
                min(256, _pow2(1.2 * width / cell)))
    cfg = dict(cellSize=cell, gridDims=dims)
    if total > 300000:
        cfg["maxPairs"] = 8 * (total + worlds)
    return cfg


def _throw(case, seed):
    """The differentiable throw: a block of cubes per world with velocities."""
    worlds, per = case["worlds"], case["bodies"]
    total = worlds * per
    local = (_lattice(per, 4) - [1.5, 0.0, 1.5]) * 1.05 + [0.0, 0.55, 0.0]
    pos = np.tile(local, (worlds, 1))
    wid = np.repeat(np.arange(worlds), per)
    f32 = np.float32
    return scenes.Scene(
        name="perf_throw", shapes=[scenes.box_vertices(10.0, 0.5, 10.0), scenes.box_vertices(0.5, 0.5, 0.5)],
        num_worlds=worlds, shape=np.concatenate([np.zeros(worlds), np.ones(total)]).astype(np.int32),
        mass=np.concatenate([np.zeros(worlds), scenes.uniform(seed, 21, total, 0.5, 2.0)]).astype(f32),
        pos=np.concatenate([_grounds(worlds, [0.0, -0.5, 0.0]), pos]).astype(f32),
        quat=np.tile([0.0, 0.0, 0.0, 1.0], (worlds + total, 1)).astype(f32),
        friction=np.concatenate([np.full(worlds, 0.6), scenes.uniform(seed, 22, total, 0.3, 0.9)]).astype(f32),
        world=np.concatenate([np.arange(worlds), wid]).astype(np.int32),
        lin=np.concatenate([np.zeros((worlds, 3)), scenes.normal(seed, 20, 3 * total, 1.0).reshape(total, 3)]).astype(f32),
        ang=np.zeros((worlds + total, 3), f32), config=dict(cellSize=1.0, gridDims=(16, 16, 16)))


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
_context = None


def _ctx():
    global _context
    if _context is None:
        torch.cuda.init()
        _context = b3.Context(torch.cuda.current_device())
    return _context


class _View:
    """A borrowed device buffer of a world, for torch.as_tensor."""

    def __init__(self, owner, which, shape, typestr):
        ptr, _ = owner.device_buffer(which)
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3)


def _views(w):
    names = ("pos", "quat", "linVel", "angVel")
    return {k: torch.as_tensor(_View(w, k, (w.n, 4), "<f4"), device="cuda") for k in names}


def _world(scene, case):
    flags = (b3.B3_WORLD_SAP_BROADPHASE if case.get("broadphase") == "sap" else 0) | \
        (b3.B3_WORLD_BATCHED_GS_SOLVER if case.get("solver") == "gs" else 0)
    w = scenes.build_world(_ctx(), scene, useGraph=1, flags=flags)
    views = _views(w)
    start = {k: v.clone() for k, v in views.items()}
    return w, views, start


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        w, views, start = _world(_scene(case, seed), case)
        counters = torch.as_tensor(_View(w, "counters", (5,), "<i4"), device="cuda")
        if case["autotune"]:
            w.autotune(3)
        return dict(kind=kind, w=w, views=views, start=start, counters=counters)
    if kind == "adjoint":
        w, views, start = _world(_throw(case, seed), case)
        adj = b3.Adjoint(w, case["steps"], case["every"])
        target = scenes.uniform(seed, 23, 3 * w.n, -3.0, 3.0).reshape(w.n, 3)
        return dict(kind=kind, w=w, adj=adj, views=views, start=start, seed_pos=target.astype(np.float32))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    if kind == "sort":
        top = 1 << case["bits"]
        keys = torch.randint(0, top, (n,), generator=gen, device="cuda", dtype=torch.int64)
        keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
        vals = torch.arange(n, device="cuda", dtype=torch.int32)
        form = case["form"]
        sort = b3.RadixSort32(_ctx())
        if form == "records":
            return dict(kind=kind, form=form, sort=sort, bits=case["bits"], records=torch.stack([keys, vals], 1).contiguous(),
                        work=torch.empty((n, 2), device="cuda", dtype=torch.int32))
        return dict(kind=kind, form=form, sort=sort, bits=case["bits"], keys=keys, vals=vals, keys_out=torch.empty_like(keys),
                    vals_out=torch.empty_like(vals))
    cells = case["cells"]
    rec = torch.stack([torch.randint(0, cells, (n,), generator=gen, device="cuda", dtype=torch.int32),
                       torch.arange(n, device="cuda", dtype=torch.int32)], 1).contiguous()
    return dict(kind=kind, cells=cells, bits=max(1, (cells - 1).bit_length()), records=rec, work=torch.empty_like(rec),
                count=torch.empty(cells, device="cuda", dtype=torch.int32),
                offset=torch.empty(cells, device="cuda", dtype=torch.int32), sort=b3.RadixSort32(_ctx()),
                search=b3.BoundSearch(_ctx()), scan=b3.PrefixScan(_ctx()))


def _reset(s):
    for k, v in s["views"].items():
        v.copy_(s["start"][k])


def run(s):
    kind = s["kind"]
    if kind == "step":
        _reset(s)
        s["w"].stepSimulation(1)
        # pairs, manifolds, contact points, and what the caps dropped
        return dict(s["views"], counts=s["counters"])
    if kind == "adjoint":
        _reset(s)
        s["adj"].forward()
        final = s["views"]["pos"].clone()
        s["adj"].backward(d_pos=s["seed_pos"])
        return dict(s["adj"].gradients(), final=final)
    if kind == "sort":
        if s["form"] == "records":  # in place, as the reference's (key, value) records are sorted
            s["work"].copy_(s["records"])
            s["sort"].execute_sortdata(s["work"], key_bits=s["bits"])
            return dict(records=s["work"])
        if s["form"] == "keys":
            s["keys_out"].copy_(s["keys"])
            s["sort"].execute(s["keys_out"], key_bits=s["bits"])
            return dict(keys=s["keys_out"])
        s["sort"].execute_out(s["keys"], s["keys_out"], s["vals"], s["vals_out"], key_bits=s["bits"])
        return dict(keys=s["keys_out"], vals=s["vals_out"])
    s["work"].copy_(s["records"])
    n = s["work"].shape[0]
    s["sort"].execute_sortdata(s["work"], key_bits=s["bits"])
    s["search"].execute_sortdata(s["work"], n, s["count"], s["cells"], b3.BoundSearch.COUNT)
    total = s["scan"].execute(s["count"], s["offset"])
    return dict(records=s["work"], count=s["count"], offset=s["offset"], total=total)


# What a body of each shape set meets on average: touching pairs, and the
# separating-axis operations of one of its pairs (axes x vertices x 5)
_TOUCH = {"cubes": 2.5, "mixed": 3.0, "hulls": 2.5, "spheres": 3.0, "compounds": 2.0, "terrain": 4.0}
_AXES = {"cubes": 15 * 16 * 5, "mixed": 60 * 40 * 5, "hulls": 40 * 20 * 5, "spheres": 10, "compounds": 30 * 20 * 5,
         "terrain": 20 * 12 * 5}


def work(case):
    kind = case["kind"]
    if kind == "sort":
        per = 4 if case["form"] == "keys" else 8
        return dict(bytes=2 * per * case["n"], flops=0)
    if kind == "cells":
        return dict(bytes=16 * case["n"] + 8 * case["cells"], flops=0)
    bodies = case["bodies"] * case["worlds"]
    # state in and out, masses, inertia, friction and shape of each body; per
    # touching pair its axis search and 10 solver iterations of 12 rows
    touch = 0.4 if case.get("packing") == "falling" else _TOUCH[case.get("shapes", "cubes")]
    flops = bodies * touch * (_AXES[case.get("shapes", "cubes")] + 10 * 12 * 40)
    nbytes = bodies * (2 * 64 + 36)
    if kind == "adjoint":  # a forward step and about twice its work in reverse
        return dict(bytes=3 * case["steps"] * nbytes, flops=3 * case["steps"] * flops)
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def exact(case, seed):
    """One step of spheres on a plane in 64 bits: gravity, contacts, Jacobi rows
    and averaging, integration. A step of polyhedra has no such short statement
    (its contacts come out of an axis search and clipping with ties decided by
    index), a throw's gradients go through several of those, and sorts, searches
    and scans give whole numbers."""
    if case["kind"] != "step" or case["shapes"] != "spheres" or case["solver"] != "jacobi":
        return None
    sc = _scene(case, seed)
    f8 = np.float64
    r = np.array([0.0] + list(_radii(seed)), f8)[sc.shape]
    dt, g, slop, erp = f8(np.float32(1 / 60)), f8(np.float32(-9.8)), f8(np.float32(0.01)), f8(np.float32(0.2))
    pos, lin, ang, quat = (a.astype(f8) for a in (sc.pos, sc.lin, sc.ang, sc.quat))
    m = sc.mass.astype(f8)
    dyn = m > 0
    im = np.where(dyn, 1.0 / np.where(dyn, m, 1.0), 0.0)
    # inertia of the registration box (radius plus its 0.01 margin), full extents doubled
    side = 2.0 * (2.0 * (r + f8(np.float32(0.01))))
    ii = np.where(dyn, 1.0 / (np.where(dyn, m, 1.0) / 12.0 * 2.0 * side * side + ~dyn), 0.0)
    lin[dyn, 1] += g * dt
    # contacts: sphere pairs (A the higher index) and the plane with each sphere
    ia, ib = _near(pos, r)
    d = pos[ia] - pos[ib]
    dist = np.linalg.norm(d, axis=1)
    n1 = d / dist[:, None]  # from B to A: minus the contact normal
    low = np.nonzero(dyn & (pos[:, 1] - r < 0.0))[0]
    A = np.concatenate([ia, np.zeros(len(low), np.int64)])
    B = np.concatenate([ib, low])
    n = np.concatenate([n1, np.tile([0.0, -1.0, 0.0], (len(low), 1))])
    depth = np.concatenate([dist - r[ia] - r[ib], pos[low, 1] - r[low]])
    point = np.concatenate([pos[ib] + n1 * r[ib][:, None], pos[low] - np.array([0.0, 1.0, 0.0]) * r[low][:, None]])
    M = len(A)
    dA, dB = dyn[A], dyn[B]
    count = np.bincount(A[dA], minlength=len(m)) + np.bincount(B[dB], minlength=len(m))
    kA, kB = np.where(dA, count[A], 1.0), np.where(dB, count[B], 1.0)
    gap = depth + slop
    r1, r2 = point + n * gap[:, None] - pos[A], point - pos[B]
    vA, vB, wA, wB = (np.where(x[:, None], y, 0.0) for x, y in ((dA, lin[A]), (dB, lin[B]), (dA, ang[A]), (dB, ang[B])))
    imA, imB, iiA, iiB = im[A], im[B], ii[A], ii[B]

    def row(axis):
        """Jacobian, effective mass, scaled one and relative velocity along axis."""
        t1, t2 = np.cross(r1, axis), np.cross(r2, -axis)
        d0 = imA + np.sum(t1 * t1, 1) * iiA
        d1 = imB + np.sum(t2 * t2, 1) * iiB
        rel = np.sum(axis * (vA - vB), 1) + np.sum(t1 * wA, 1) + np.sum(t2 * wB, 1)
        return [axis, t1, t2, 1.0 / (d0 + d1), 1.0 / (d0 * kA + d1 * kB), rel]

    normal = row(n)
    push = np.where(gap > 0.0, -gap / dt, -gap * erp / dt)
    rhs_n = (push - normal[5]) * normal[4]
    vel = vA + np.cross(wA, r1) - vB - np.cross(wB, r2)
    along = np.sum(n * vel, 1)
    t = vel - n * along[:, None]
    lat = np.sum(t * t, 1)
    slide = lat > np.finfo(np.float32).eps
    p, q = _tangents(n)
    u1 = np.where(slide[:, None], t / np.sqrt(np.where(slide, lat, 1.0))[:, None], p)
    u2 = np.cross(u1, n)
    u2 = np.where(slide[:, None], u2 / np.maximum(np.linalg.norm(u2, axis=1), 1e-300)[:, None], q)
    rows_f = [row(u2), row(u1)]
    mu = np.sqrt(sc.friction.astype(f8)[A] * sc.friction.astype(f8)[B])
    lam_n, lam_f = np.zeros(M), [np.zeros(M), np.zeros(M)]
    avg_v, avg_w = np.zeros_like(pos), np.zeros_like(pos)

    def solve(rw, rhs, lam, lo, hi, dv, on):
        axis, t1, t2, eff = rw[0], rw[1], rw[2], rw[3]
        rel = np.sum(axis * (dv[0] - dv[2]), 1) + np.sum(t1 * dv[1], 1) + np.sum(t2 * dv[3], 1)
        new = np.where(on, np.clip(lam + rhs - rel * eff, lo, hi), lam)
        delta = (new - lam)[:, None]
        dv[0] += axis * imA[:, None] * delta
        dv[1] += t1 * iiA[:, None] * delta
        dv[2] -= axis * imB[:, None] * delta
        dv[3] += t2 * iiB[:, None] * delta
        return new

    for _ in range(10):
        for friction in (False, True):
            dv = [np.where(dA[:, None], avg_v[A], 0.0), np.where(dA[:, None], avg_w[A], 0.0),
                  np.where(dB[:, None], avg_v[B], 0.0), np.where(dB[:, None], avg_w[B], 0.0)]
            if friction:
                on, lim = lam_n > 0.0, mu * lam_n
                for k in (0, 1):
                    lam_f[k] = solve(rows_f[k], -rows_f[k][5] * rows_f[k][4], lam_f[k], -lim, lim, dv, on)
            else:
                lam_n = solve(normal, rhs_n, lam_n, 0.0, 1e10, dv, True)
            for out, xa, xb in ((avg_v, dv[0], dv[2]), (avg_w, dv[1], dv[3])):
                out[:] = 0.0
                np.add.at(out, A[dA], xa[dA])
                np.add.at(out, B[dB], xb[dB])
                out /= np.maximum(count, 1)[:, None]
    # every copy of a body adds the average, then damping and integration
    lin += avg_v * count[:, None]
    ang = np.where(dyn[:, None], (ang + avg_w * count[:, None]) * f8(np.float32(0.99)), ang)
    angle = np.minimum(np.linalg.norm(ang, axis=1), 0.25 * math.pi / dt)
    small = angle < 0.001
    s = np.where(small, 0.5 * dt - dt ** 3 * 0.020833333333 * angle * angle,
                 np.sin(0.5 * angle * dt) / np.where(small, 1.0, angle))
    dq = np.concatenate([ang * s[:, None], np.cos(0.5 * angle * dt)[:, None]], 1)
    turned = np.concatenate([dq[:, 3:] * quat[:, :3] + quat[:, 3:] * dq[:, :3] + np.cross(dq[:, :3], quat[:, :3]),
                             (dq[:, 3] * quat[:, 3] - np.sum(dq[:, :3] * quat[:, :3], 1))[:, None]], 1)
    turned /= np.linalg.norm(turned, axis=1, keepdims=True)
    zero = np.zeros((len(m), 1))
    return dict(pos=np.concatenate([np.where(dyn[:, None], pos + lin * dt, pos), zero], 1),
                quat=np.where(dyn[:, None], turned, quat), linVel=np.concatenate([lin, zero], 1),
                angVel=np.concatenate([ang, zero], 1), counts=None)


def _near(pos, r):
    """Touching sphere pairs (higher index first), by 1 m cells."""
    body = np.nonzero(r > 0)[0]
    c = np.floor(pos[body]).astype(np.int64) + 4096
    key = (c[:, 0] * 8192 + c[:, 1]) * 8192 + c[:, 2]
    order = np.argsort(key, kind="stable")
    skey = key[order]
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                want = key + (dx * 8192 + dy) * 8192 + dz
                lo, hi = np.searchsorted(skey, want, "left"), np.searchsorted(skey, want, "right")
                for k in range(int((hi - lo).max()) if len(lo) else 0):
                    i = np.nonzero(lo + k < hi)[0]
                    j = order[lo[i] + k]
                    a, b = body[i], body[j]
                    keep = (a > b) & (np.sum((pos[a] - pos[b]) ** 2, 1) <= (r[a] + r[b]) ** 2)
                    found.append((a[keep], b[keep]))
    return np.concatenate([f[0] for f in found]), np.concatenate([f[1] for f in found])


def _tangents(n):
    """Two unit vectors across n, by the larger of its components."""
    z = np.abs(n[:, 2]) > 0.7071067811865475
    a = np.where(z, n[:, 1] ** 2 + n[:, 2] ** 2, n[:, 0] ** 2 + n[:, 1] ** 2)
    k = 1.0 / np.sqrt(a)
    o = np.zeros(len(n))
    p = np.where(z[:, None], np.stack([o, -n[:, 2] * k, n[:, 1] * k], 1), np.stack([-n[:, 1] * k, n[:, 0] * k, o], 1))
    q = np.where(z[:, None], np.stack([a * k, -n[:, 0] * p[:, 2], n[:, 0] * p[:, 1]], 1),
                 np.stack([-n[:, 2] * p[:, 1], n[:, 2] * p[:, 0], a * k], 1))
    return p, q
