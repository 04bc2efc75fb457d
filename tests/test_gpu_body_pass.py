"""The solve with a pass over the bodies (k_jacobi_pass) at sizes from a few dozen
manifolds on. Up to 524,288 expected manifolds (three per body) both forms are
launched, and the device takes the one with rows in shared memory while there are
no more than expected, rounded up to 64; cubes pressed into each other, 26
neighbours each, have more, so that the pass runs. Its steps are those of the other
form, value for value, whatever the CTA size and the blocks per SM."""
import numpy as np
import pytest

from experiments_b200 import scenes

pytestmark = pytest.mark.gpu


def pressed(side, more=0):
    n = side ** 3 + more
    i = np.arange(n)
    pos = np.stack([(i % side) * 0.6, 0.48 + (i // (side * side)) * 0.6, (i // side % side) * 0.6], 1)
    pos += scenes.uniform(7, 1, 3 * n, -0.01, 0.01).reshape(n, 3)
    b = scenes._concat([scenes.ground(), scenes._bodies(np.ones(n, np.int32), scenes.uniform(7, 2, n, 0.5, 2.0), pos,
                                                        scenes.yaw_quat(scenes.uniform(7, 3, n, 0.0, 0.3)),
                                                        np.full(n, 0.6), np.zeros(n, np.int32),
                                                        lin=scenes.normal(7, 4, 3 * n, 0.3).reshape(n, 3))])
    return scenes.Scene(name="pressed", shapes=[scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5)],
                        num_worlds=1, config=dict(cellSize=1.0, gridDims=(16, 16, 16), maxBodiesPerCell=256), **b)


@pytest.mark.parametrize("side,more", [(3, 0), (4, 0), (4, 3), (5, 0), (5, 11), (10, 0), (14, 37)])
def test_pass_over_the_bodies_at_small_sizes(ctx, side, more):
    sc = pressed(side, more)
    states = []
    for gather, threads, cap in ((0, 64, 4), (1, 64, 1), (1, 128, 2), (1, 256, 4), (1, 256, 8)):
        w = scenes.build_world(ctx, sc, maxPairsPerBody=64)
        t = w.tuning()
        w.set_tuning([t[0], t[1], threads, t[3], cap, t[5], 0, gather])
        w.stepSimulation(1)
        # more than the shared memories are sized for: gather = 1 takes the pass
        assert w.counters()["numManifolds"] > (3 * sc.n + 63) // 64 * 64
        states.append(w.read_state())
        w.stepSimulation(2)
        states[-1] += w.read_state()
        assert w.counters()["timeouts"] == 0
        w.close()
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)
