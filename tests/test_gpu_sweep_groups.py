"""The lane-group sweep (pairs of few axes: boxes, mesh triangles) gives the
oracle's contacts: pair counts around a group's and a warp's size, boxes of
every proportion, pairs of both sweeps in one list, and pairs the narrowphase
skips in between."""
import numpy as np
import pytest

from experiments_b200 import scenes

from helpers import make_pair

pytestmark = pytest.mark.gpu

POS_TOL = 1e-5
NRM_TOL = 1e-4

TETRA = 0.6 * np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], np.float32)


def _heap(kind, n, seed=91):
    """Bodies turned every way on a jittered grid, each touching a few others."""
    boxes = [scenes.box_vertices(*h) for h in ((0.5, 0.5, 0.5), (0.7, 0.3, 0.5), (0.9, 0.15, 0.2), (0.6, 0.6, 0.1),
                                               (0.35, 0.35, 0.35))]
    extra = {"boxes": [], "both": [TETRA, scenes.icosphere_vertices(0.5)] + scenes.hull_pool(5, 3),
             "skipped": [{"kind": "sphere", "radius": 0.5}, {"kind": "sphere", "radius": 0.4}]}[kind]
    shapes = [scenes.box_vertices(20.0, 0.5, 20.0)] + boxes + extra
    side = max(1, int(np.ceil(n ** (1 / 3))))
    i = np.arange(n)
    pos = 0.8 * np.stack([i % side, i // (side * side), i // side % side], 1) + [0.0, 0.45, 0.0]
    pos += scenes.uniform(seed, 1, 3 * n, -0.1, 0.1).reshape(n, 3)
    q = scenes.normal(seed, 2, 4 * n).reshape(n, 4)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    sid = 1 + (scenes.uniform(seed, 3, n) * (len(shapes) - 1)).astype(int)
    b = scenes._concat([scenes.ground(), scenes._bodies(sid, np.ones(n), pos, q, np.full(n, 0.6), np.zeros(n))])
    return scenes.Scene(name="heap", shapes=shapes, num_worlds=1,
                        config=dict(cellSize=1.0, gridDims=(16, 16, 16), maxPairs=max(4096, 64 * n)), **b)


def _compare(w, o, least):
    for s in ("aabbs", "broadphase", "narrowphase"):
        w.stage(s)
    o.stage("aabbs")
    o.set_pairs(w.pairs())
    o.stage("narrowphase")
    gc, oc = w.contacts(), o.contacts()
    gi = {int(p): k for k, p in enumerate(gc["pairIndex"])}
    oi = {int(p): k for k, p in enumerate(oc["pairIndex"])}
    assert set(gi) == set(oi) and len(gi) >= least
    for p, kg in gi.items():
        ko = oi[p]
        n = int(gc["normal"][kg][3])
        assert n == int(oc["normal"][ko][3])
        assert np.abs(gc["normal"][kg][:3] - oc["normal"][ko][:3]).max() <= NRM_TOL
        assert np.abs(gc["pos"][kg][:n] - oc["pos"][ko][:n]).max() <= POS_TOL


@pytest.mark.parametrize("kind,n", [("boxes", 1), ("boxes", 2), ("boxes", 9), ("boxes", 40), ("boxes", 300),
                                    ("both", 12), ("both", 250), ("skipped", 120)])
def test_contacts_match_oracle(ctx, kind, n):
    w, o = make_pair(ctx, _heap(kind, n))
    _compare(w, o, 1 if n > 2 else 0)
    o.close()
    w.close()


def test_many_pairs_per_grab(ctx):
    """Enough pairs for 32 to a grab: the steps of a large lattice agree with
    those of its blocks stepped alone (bodies of different blocks far apart)."""
    one = scenes.c1(dims=(24, 12, 24))
    k, shift = 16, 60.0
    cat = lambda f: np.concatenate([getattr(one, f)[1:]] * k)  # noqa: E731
    pos = np.concatenate([one.pos[1:] + np.array([shift * (j % 4 - 1.5), 0, shift * (j // 4 - 1.5)], np.float32)
                          for j in range(k)])
    first = {f: getattr(one, f)[:1] for f in ("shape", "mass", "pos", "quat", "friction", "world", "lin", "ang")}
    shapes = [scenes.box_vertices(300.0, 0.5, 300.0)] + list(one.shapes[1:])
    big = scenes.Scene(name="blocks", shapes=shapes, num_worlds=1, config=dict(cellSize=1.0, gridDims=(256, 32, 256)),
                       pos=np.concatenate([first["pos"], pos]),
                       **{f: np.concatenate([first[f], cat(f)]) for f in first if f != "pos"})
    w = scenes.build_world(ctx, big, useGraph=1)
    w.stepSimulation(8)
    c = w.counters()
    w.close()
    assert c["numPairs"] > 2 * 32 * 148 * 20 and c["pairOverflow"] == 0
    per = []
    for j in range(k):
        sub = scenes.Scene(name="block", shapes=shapes, num_worlds=1,
                           config=dict(cellSize=1.0, gridDims=(256, 32, 256)),
                           pos=np.concatenate([first["pos"], pos[j * (one.n - 1):(j + 1) * (one.n - 1)]]),
                           **{f: getattr(one, f) for f in first if f != "pos"})
        v = scenes.build_world(ctx, sub)
        v.stepSimulation(8)
        per.append(v.counters())
        v.close()
    for f in ("numPairs", "numManifolds", "numContactPoints"):
        assert c[f] == sum(p[f] for p in per), f


@pytest.mark.parametrize("gap", [-0.01, 0.0, 2e-6, 0.05])
def test_pairs_left_out_before_the_sweep(ctx, gap):
    """Pairs that the sorting finds to be apart: the same cubes give the same bits
    alone, where their pairs are not sorted, and with a far icosphere beside them,
    with which they are."""
    n = 2000
    i = np.arange(n)
    side = 13
    pos = np.stack([i % side, i // (side * side), i // side % side], 1) * (1.0 + gap) + [3.0, 0.5 + gap, 3.0]
    turned = (i % 3 > 0)[:, None]
    pos = pos + np.where(turned, scenes.uniform(3, 1, 3 * n, -0.02, 0.02).reshape(n, 3), 0.0)
    quat = np.where(turned, scenes.yaw_quat(scenes.uniform(3, 2, n, 0.0, 0.8)), [0.0, 0.0, 0.0, 1.0])
    boxes = [scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5)]
    states = []
    for extra in (0, 1):
        m = n + extra
        p = np.concatenate([pos, [[50.0, 30.0, 50.0]]])[:m]
        q = np.concatenate([quat, [[0.0, 0.0, 0.0, 1.0]]])[:m]
        sid = np.append(np.ones(n, np.int32), 2)[:m]
        b = scenes._concat([scenes.ground(), scenes._bodies(sid, np.ones(m), p, q, np.full(m, 0.6), np.zeros(m))])
        w = scenes.build_world(ctx, scenes.Scene(name="beside", shapes=boxes + [scenes.icosphere_vertices(0.5)] * extra,
                                                 num_worlds=1, config=dict(cellSize=1.0, gridDims=(64, 64, 64)), **b))
        w.stepSimulation(3)
        c = w.counters()
        states.append(([a[:n + 1].copy() for a in w.read_state()], c["numManifolds"], c["refinedAxes"]))
        w.close()
    assert states[0][1:] == states[1][1:]
    for x, y in zip(states[0][0], states[1][0]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [8192, 16500])
def test_sorted_by_size(ctx, n):
    """One kind of pairs, where the bodies are just not enough for the sorting and
    where the pairs are: the same bits as with an icosphere beside them."""
    side = 26
    i = np.arange(n)
    pos = np.stack([i % side, i // (side * side), i // side % side], 1) * [1.01, 0.995, 1.01] + [3.0, 0.5, 3.0]
    pos += scenes.uniform(4, 1, 3 * n, -0.01, 0.01).reshape(n, 3)
    quat = scenes.yaw_quat(scenes.uniform(4, 2, n, 0.0, 0.3))
    boxes = [scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5)]
    states = []
    for extra in (0, 1):
        m = n + extra
        p = np.concatenate([pos, [[50.0, 50.0, 50.0]]])[:m]
        q = np.concatenate([quat, [[0.0, 0.0, 0.0, 1.0]]])[:m]
        sid = np.append(np.ones(n, np.int32), 2)[:m]
        b = scenes._concat([scenes.ground(), scenes._bodies(sid, np.ones(m), p, q, np.full(m, 0.6), np.zeros(m))])
        w = scenes.build_world(ctx, scenes.Scene(name="sorted", shapes=boxes + [scenes.icosphere_vertices(0.5)] * extra,
                                                 num_worlds=1, config=dict(cellSize=1.0, gridDims=(64, 64, 64)), **b))
        w.stepSimulation(2)
        c = w.counters()
        states.append(([a[:n + 1].copy() for a in w.read_state()], c["numPairs"], c["numManifolds"]))
        w.close()
    assert states[0][1:] == states[1][1:]
    assert states[0][1] > (51200 if n > 8192 else 0)
    for x, y in zip(states[0][0], states[1][0]):
        assert np.array_equal(x, y)
