"""The reverse sweep's forms give the same bits: rows kept in shared memory or
streamed, and a second backward pass from the states the first one left."""
import numpy as np
import pytest

from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = b3.Context(0)
    yield c
    c.close()


def _block(side, far):
    """Cubes in a lattice that overlap their 26 neighbours a little, and `far`
    cubes of the same kind that touch nothing: the launch is sized by the number
    of bodies, so without them most of the manifolds are streamed."""
    n = side ** 3
    i = np.arange(n)
    pos = np.stack([i % side, i // (side * side), i // side % side], 1) * 0.99 + [2.0, 0.49, 2.0]
    pos += scenes.uniform(9, 1, 3 * n, -0.002, 0.002).reshape(n, 3)
    k = np.arange(far)
    pos = np.concatenate([pos, np.stack([20.0 + 1.5 * (k % 24), 5.0 + 1.5 * (k // 576), 20.0 + 1.5 * (k // 24 % 24)], 1)])
    m = n + far
    quat = np.tile([0.0, 0.0, 0.0, 1.0], (m, 1))
    b = scenes._concat([scenes.ground(), scenes._bodies(np.ones(m, np.int32), np.ones(m), pos, quat, np.full(m, 0.6),
                                                        np.zeros(m))])
    lin = np.zeros((m + 1, 3), np.float32)
    lin[1:n + 1] = scenes.normal(9, 2, 3 * n, 0.1).reshape(n, 3)
    shapes = [scenes.box_vertices(100.0, 0.5, 100.0), scenes.box_vertices(0.5, 0.5, 0.5)]
    b["lin"] = lin
    return scenes.Scene(name="block", shapes=shapes, num_worlds=1, config=dict(cellSize=1.0, gridDims=(64, 16, 64)), **b), n


def _gradients(ctx, sc, n, steps, every, times=1):
    w = scenes.build_world(ctx, sc)
    adj = b3.Adjoint(w, steps, every)
    adj.forward()
    seed = np.zeros((w.n, 3), np.float32)
    seed[1:n + 1] = scenes.uniform(9, 3, 3 * n, -1.0, 1.0).reshape(n, 3)
    out = []
    for _ in range(times):
        adj.backward(d_pos=seed, d_lin=seed)
        g = adj.gradients()
        state = [a[:n + 1].copy() for a in w.read_state()]
        out.append([g[k][:n + 1].copy() for k in ("lin", "ang", "mass", "friction")] + state)
    c = w.counters()
    adj.close()
    w.close()
    return out, c


# a few manifolds; more than a CTA; with and without a remainder of streamed ones
@pytest.mark.parametrize("side", [1, 3, 4, 5])
def test_streamed_rows_give_the_same_bits(ctx, side):
    near, n = _block(side, 0)
    wide, _ = _block(side, 2000)
    (a,), ca = _gradients(ctx, near, n, 1, 1)
    (b,), cb = _gradients(ctx, wide, n, 1, 1)
    assert ca["numManifolds"] == cb["numManifolds"] > 0
    if side >= 4:  # above the threads launched for so few bodies
        blocks = -(-3 * (n + 1) // 128)
        assert ca["numManifolds"] > 128 * blocks
    for x, y in zip(a, b):
        assert np.isfinite(x).all() and np.array_equal(x, y)


@pytest.mark.parametrize("steps,every", [(1, 1), (5, 5), (5, 2), (4, 2)])
def test_backward_repeats(ctx, steps, every):
    sc, n = _block(3, 0)
    (a, b), _ = _gradients(ctx, sc, n, steps, every, times=2)
    (c,), _ = _gradients(ctx, sc, n, steps, 1)
    for x, y, z in zip(a, b, c):
        assert np.array_equal(x, y) and np.array_equal(x, z)
