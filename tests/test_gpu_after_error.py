"""Steps between a wait that gave up and the host's reset of it.

The world keeps its error flag until b3_reset_counters, and a caller may step
on before it looks. Those steps' results are void, but they have to stay within
their buffers: the sorts run whatever the flag holds (their output is what the
contact list, the solve and the pair search index with), and after the reset
and a written state the world steps like a new one, bit for bit.
"""
import numpy as np
import pytest

from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu

B3_ERR_TIMEOUT = 6


def cubes(side, gap):
    """side^3 unit cubes over the ground, layers `gap` apart (0.995: every layer
    rests on the one below; 1.05: only the lowest touches)."""
    n = side ** 3
    i = np.arange(n)
    pos = np.stack([(i % side) * 1.05, 0.495 + (i // (side * side)) * gap, (i // side % side) * 1.05], 1)
    pos[:, [0, 2]] -= 0.525 * (side - 1)
    quat = np.tile([0.0, 0.0, 0.0, 1.0], (n, 1))
    b = scenes._concat([scenes.ground(), scenes._bodies(np.ones(n, np.int32), np.ones(n), pos, quat, np.full(n, 0.6),
                                                        np.zeros(n, np.int32))])
    return scenes.Scene(name="cubes", shapes=[scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5)],
                        num_worlds=1, config=dict(cellSize=1.0, gridDims=(64, 64, 64)), **b)


def state(sc):
    n = sc.n
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = sc.pos
    return pos, np.asarray(sc.quat, np.float32), np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)


@pytest.mark.parametrize("side,flags", [(6, 0), (22, 0), (41, 0), (22, b3.B3_WORLD_SAP_BROADPHASE)])
def test_steps_after_a_wait_gave_up_stay_in_bounds(ctx, side, flags):
    """The solve's barrier gives up while few bodies touch; steps follow with far
    more contacts than any before. 216 and 68,921 bodies: body numbers of one and
    three digits, whose sort ends in the other buffer; 10,648: of two."""
    few, many = cubes(side, 1.05), cubes(side, 0.995)
    cap = max(8192, 16 * few.n)  # sorts of more than one block
    w = scenes.build_world(ctx, few, maxPairs=cap, flags=flags)
    t = w.tuning()
    t = [t[0], t[1], 64, t[3], 4, t[5], 0, t[7]]  # many blocks in the solve
    w.set_tuning(t)
    w.stepSimulation(2)
    rc, c = w.counters_status()
    assert rc == 0 and 0 < c["numManifolds"] <= side * side
    w.set_wait_limits(spin_limit=8, hold_micros=20000)
    w.write_state(*state(few))
    w.stepSimulation(1)
    rc, c = w.counters_status()
    assert rc == B3_ERR_TIMEOUT and c["timeouts"] > 0
    w.write_state(*state(many))
    w.stepSimulation(1)
    rc, c = w.counters_status()
    assert rc == B3_ERR_TIMEOUT and c["numManifolds"] > 2 * side * side
    w.stepSimulation(2)
    w.set_wait_limits()
    w.reset_counters()
    fresh = scenes.build_world(ctx, few, maxPairs=cap, flags=flags)
    fresh.set_tuning(t)
    for sc in (many, few):
        for x in (w, fresh):
            x.write_state(*state(sc))
            x.stepSimulation(2)
            rc, c = x.counters_status()
            assert rc == 0 and c["timeouts"] == 0
        for a, b in zip(w.read_state(), fresh.read_state()):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    w.close()
    fresh.close()
