"""A new world on a stream of the caller's while the default stream is busy: the
clears of its buffers (the cell table, the scalars, the sorts' buffers and barrier
words) are done before it steps, and it steps as any other world."""
import numpy as np
import pytest

from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 9000])
def test_new_world_steps_on_its_stream_while_the_default_stream_is_busy(ctx, n):
    import torch
    sc = scenes.random_pile(91, n=n, box=2.0 * n ** (1 / 3), hull_frac=0.3)
    states = []
    for busy in (False, True):
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        if busy:
            torch.cuda._sleep(100_000_000)  # some 50 ms on the default stream
        w = b3.PhysicsWorld(ctx, scenes.world_config(sc))
        scenes.register_scene(w, sc)
        w.writeBodiesToGpu(stream=stream.cuda_stream)
        w.stepSimulation(4, stream=stream.cuda_stream)
        states.append(w.read_state(stream=stream.cuda_stream))
        assert w.counters()["timeouts"] == 0
        w.close()
    for a, b in zip(*states):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
