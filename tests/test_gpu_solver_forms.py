"""The Jacobi solve's forms give the same bits: averages gathered by every
manifold with rows kept in shared memory, averages formed by a pass over the
bodies, and one block per world, at the sizes where they take other paths."""
import numpy as np
import pytest

from experiments_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from experiments_b200 import b3
    c = b3.Context(0)
    yield c
    c.close()


def _heap(n, plate):
    """Cubes in touching layers; with `plate`, a dynamic slab under them that
    touches far more bodies than one round of loads takes."""
    side = max(2, int(round((2.0 * n) ** (1 / 3))))
    i = np.arange(n)
    pos = np.stack([(i % side) * 1.02, 0.49 + (i // (side * side)) * 0.99, (i // side % side) * 1.02], 1)
    pos += scenes.uniform(7, 1, 3 * n, -0.01, 0.01).reshape(n, 3)
    quat = scenes.yaw_quat(scenes.uniform(7, 2, n, 0.0, 0.4))
    shapes = [scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5),
              scenes.box_vertices(20.0, 0.25, 20.0)]
    sid, mass = np.ones(n, np.int32), scenes.uniform(7, 3, n, 0.5, 2.0)
    if plate:
        pos[:, 1] += 0.49
        pos = np.concatenate([pos, [[side / 2, 0.24, side / 2]]])
        quat = np.concatenate([quat, [[0, 0, 0, 1.0]]])
        sid, mass = np.append(sid, 2), np.append(mass, 50.0)
    b = scenes._concat([scenes.ground(), scenes._bodies(sid, mass, pos, quat, scenes.uniform(7, 4, len(sid), 0.3, 0.9),
                                                        np.zeros(len(sid)))])
    return scenes.Scene(name="heap", shapes=shapes, num_worlds=1, config=dict(cellSize=1.0, gridDims=(64, 64, 64)), **b)


def _run(ctx, sc, threads, cap, mode, form, steps=4):
    w = scenes.build_world(ctx, sc, useGraph=1)
    t = w.tuning()
    w.set_tuning([t[0], t[1], threads, t[3], cap, t[5], mode, form])
    w.stepSimulation(steps)
    out = w.read_state()
    c = w.counters()
    w.close()
    return out, c


# one manifold; under and over one CTA; a body with hundreds of copies; more
# manifolds than 64-thread CTAs keep in shared memory, the rest streamed
@pytest.mark.parametrize("n,plate", [(1, False), (20, False), (300, True), (9000, False), (24000, False), (24000, True)])
def test_forms_give_the_same_bits(ctx, n, plate):
    sc = _heap(n, plate)
    ref, c = _run(ctx, sc, 256, 4, 0, 1)
    assert c["numManifolds"] > 0 and c["pairOverflow"] == 0
    for threads, cap in ((64, 1), (64, 8), (256, 1)):
        got, g = _run(ctx, sc, threads, cap, 0, 0)
        assert g == c
        for a, b in zip(ref, got):
            assert np.array_equal(a, b)


def test_worlds_give_the_same_bits(ctx):
    sc = scenes.random_pile(44, n=40, worlds=9, hull_frac=0.5)
    ref, _ = _run(ctx, sc, 128, 4, 0, 1)
    for mode, form in ((0, 0), (1, 0), (1, 1)):
        got, _ = _run(ctx, sc, 64, 4, mode, form)
        for a, b in zip(ref, got):
            assert np.array_equal(a, b)


def test_untuned_shapes_follow_the_body_count(ctx):
    small = scenes.build_world(ctx, _heap(20, False))
    assert small.tuning()[7] == 0 and small.tuning()[2] == 64
    small.close()
    large = scenes.build_world(ctx, _heap(24000, False))
    assert large.tuning()[7] == 1 and large.tuning()[2] == 128
    t = large.tuning()
    large.set_tuning([t[0], t[1], 256, t[3], 2, t[5], 0, 0])
    large.writeBodiesToGpu()
    assert large.tuning()[2] == 256 and large.tuning()[7] == 0
    large.close()
