"""Many contacts of one dynamic body in the batched Gauss-Seidel solver.

A body's contacts in one parity class take one batch each, up to 1,024; past the
63 that one word holds they are in a set of their own. Unit cubes 4 m apart lie on
a dynamic plate, all in cells of the same class, so that the number on a plate is
the length of its run; the batches are those of the sequential greedy pass.
"""
import numpy as np
import pytest

from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu
GS = b3.B3_WORLD_BATCHED_GS_SOLVER
B3_ERR_TIMEOUT = 6


def plates(counts, extra=0, gap=-0.005):
    """One plate per count, side by side in x, each overlapping the next by 5 cm,
    with that many cubes on it (`gap` above it); `extra` cubes in the air."""
    side = int(np.ceil(np.sqrt(max(counts))))
    half = 2.0 * side + 0.025
    pos, sid, mass = [], [], []
    for k, n in enumerate(counts):
        i = np.arange(n)
        x0 = 4.0 * side * k
        pos.append(np.stack([x0 + 4.0 * (i % side) + 1.0, np.full(n, 1.0 + gap), 4.0 * (i // side) + 1.0], 1))
        sid += [1] * n
        mass += [1.0] * n
    for k in range(len(counts)):
        pos.append([[4.0 * side * k + 2.0 * side, 0.25, 2.0 * side]])
        sid.append(2)
        mass.append(80.0)
    if extra:
        i = np.arange(extra)
        pos.append(np.stack([(i % 64) * 2.0, 20.0 + (i // 4096) * 2.0, (i // 64 % 64) * 2.0], 1))
        sid += [1] * extra
        mass += [1.0] * extra
    pos = np.concatenate(pos)
    n = len(pos)
    b = scenes._concat([scenes.ground(size=2000.0), scenes._bodies(np.array(sid, np.int32), np.array(mass), pos,
                                                                   np.tile([0.0, 0.0, 0.0, 1.0], (n, 1)), np.full(n, 0.6),
                                                                   np.zeros(n, np.int32))])
    return scenes.Scene(name="plates", shapes=[scenes.box_vertices(1000.0, 0.5, 1000.0), scenes.box_vertices(0.5, 0.5, 0.5),
                                               scenes.box_vertices(half, 0.25, half)],
                        num_worlds=1, config=dict(cellSize=2.0, gridDims=(128, 32, 64)), **b)


def greedy(sc, g, c):
    """Batches of the sequential pass in (class, cell, manifold) order: the lowest
    that no earlier manifold on the same dynamic bodies of the class has."""
    dyn = np.asarray(sc.mass) > 0
    cls = (g[:, 0] & 1) + 2 * ((g[:, 0] // 16) & 1)
    seen, want = {}, np.full(len(g), -1)
    for m in np.lexsort((np.arange(len(g)), g[:, 0], cls)):
        bodies = [(int(cls[m]), x) for x in (abs(int(c["bodyA"][m])), abs(int(c["bodyB"][m]))) if dyn[x]]
        taken = set().union(*[seen.get(x, set()) for x in bodies]) if bodies else set()
        want[m] = next(k for k in range(len(taken) + 1) if k not in taken)
        for x in bodies:
            seen.setdefault(x, set()).add(int(want[m]))
    return want


@pytest.mark.parametrize("counts", [(62,), (63,), (64,), (65,), (128, 40), (63, 64, 200), (320, 700), (1024,)])
def test_batches_of_long_runs_are_the_sequential_ones(ctx, counts):
    sc = plates(counts)
    w = scenes.build_world(ctx, sc, flags=GS)
    for s in ("aabbs", "broadphase", "narrowphase", "solve"):
        w.stage(s)
    rc, n = w.counters_status()
    g, c = w.gs_batches(), w.contacts()
    assert rc == 0 and len(g) == len(c["bodyA"]) >= sum(counts)
    assert np.array_equal(g[:, 1], greedy(sc, g, c))
    assert g[:, 1].max() >= max(counts) - 1
    w.close()


@pytest.mark.parametrize("extra", [0, 66000])
def test_more_batches_than_there_are_and_the_steps_after(ctx, extra):
    """1,089 contacts of one class on a plate are more than 1,024 batches: an error.
    Steps that follow before the reset make no use of what was not coloured (with
    66,000 more bodies the entries' sort ends in its other buffer), and after it the
    world steps like a new one."""
    few, many = plates((1089,), extra, 0.5), plates((1089,), extra)
    state = lambda sc: (np.concatenate([sc.pos, np.zeros((sc.n, 1))], 1).astype(np.float32), sc.quat.astype(np.float32),
                        np.zeros((sc.n, 4), np.float32), np.zeros((sc.n, 4), np.float32))
    w = scenes.build_world(ctx, few, flags=GS)
    w.stepSimulation(2)
    assert w.counters_status()[0] == 0
    w.write_state(*state(many))
    w.stepSimulation(1)
    rc, c = w.counters_status()
    assert rc == B3_ERR_TIMEOUT and c["numManifolds"] >= 1089
    w.stepSimulation(2)
    assert w.counters_status()[0] == B3_ERR_TIMEOUT
    w.reset_counters()
    fresh = scenes.build_world(ctx, few, flags=GS)
    for x in (w, fresh):
        x.write_state(*state(few))
        x.stepSimulation(3)
        assert x.counters_status()[0] == 0
    for a, b in zip(w.read_state(), fresh.read_state()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    w.close()
    fresh.close()
