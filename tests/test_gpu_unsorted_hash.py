"""b3_get_sorted_hash between b3_stage_aabbs and b3_stage_broadphase: this step's
keys in body order, whichever buffer the sort will read them from; after the
broadphase, the same keys sorted."""
import numpy as np
import pytest

from experiments_b200 import scenes

pytestmark = pytest.mark.gpu


# 64 x 32 x 64 cells: keys of 17 bits, three passes; 16^3 cells: two; up to 8,192
# bodies are sorted in place
@pytest.mark.parametrize("n,dims", [(300, (64, 32, 64)), (9000, (64, 32, 64)), (9000, (16, 16, 16)), (70000, (64, 32, 64))])
def test_keys_before_and_after_the_sort(ctx, n, dims):
    sc = scenes.random_pile(31, n=n, box=1.2 * n ** (1 / 3), hull_frac=0.0)
    w = scenes.build_world(ctx, sc, gridDims=dims)
    w.stepSimulation(2)
    for _ in range(2):
        w.stage("aabbs")
        k0, v0 = w.sorted_hash()
        small = len(k0)
        assert np.array_equal(v0, np.arange(w.n - small, w.n))  # the ground is the one large body
        w.stage("broadphase")
        k1, v1 = w.sorted_hash()
        order = np.argsort(k0, kind="stable")
        assert np.array_equal(k1, k0[order]) and np.array_equal(v1, v0[order])
        assert len(np.unique(k1)) > 10
        pos, quat, lin, ang = w.read_state()
        pos[:, :3] += 1.7  # other cells the next time
        w.write_state(pos, quat, lin, ang)
    w.close()


def test_keys_after_a_replayed_step(ctx):
    """A captured step that follows b3_stage_aabbs sorts its own keys."""
    sc = scenes.random_pile(32, n=9000, box=60.0, hull_frac=0.0)  # cells of all three digits
    hashes = []
    for staged in (False, True):
        w = scenes.build_world(ctx, sc, gridDims=(64, 32, 64), useGraph=1)
        w.stepSimulation(2)
        state = w.read_state()
        if staged:
            w.stage("aabbs")
            w.write_state(*state)
        w.stepSimulation(1)
        hashes.append(w.sorted_hash())
        w.close()
    for a, b in zip(*hashes):
        assert np.array_equal(a, b)
    assert np.all(np.diff(hashes[0][0].astype(np.int64)) >= 0)
