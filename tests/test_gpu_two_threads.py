"""Host threads that step worlds of their own on one device. The solves of these
worlds keep different amounts of rows in shared memory, and every launch has to go
through whichever thread launched last. The threads run in C, where nothing makes
them take turns."""
import ctypes as C
import subprocess
import threading

import numpy as np
import pytest

from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu

LOOP = """
typedef int (*call_t)(void*, void*);
typedef int (*sync_t)(void*);
int loop(call_t f, sync_t sync, void* world, void* stream, int n, int each, volatile int* stop) {
    for (int i = 0; i < n && !*stop; ++i) {
        const int rc = f(world, stream);
        if (rc) { *stop = rc; return rc; }
        if (i % each == each - 1) sync(stream);
    }
    sync(stream);
    return 0;
}
"""


def _world(ctx, n):
    w = scenes.build_world(ctx, scenes.c1(dims=(n, n, n)), useGraph=0)
    t = w.tuning()
    w.set_tuning([t[0], t[1], 256, t[3], 1, t[5], 0, 0])  # one block of 256 on each SM
    w.stepSimulation(3)
    return w


def test_solves_of_three_worlds_on_three_threads(ctx, tmp_path):
    import torch
    src, so = tmp_path / "loop.c", tmp_path / "loop.so"
    src.write_text(LOOP)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    loop = C.CDLL(str(so)).loop
    sync = C.CDLL("libcudart.so.12").cudaStreamSynchronize
    # 513 and 730 bodies: one manifold of each thread kept; 10,649: two
    worlds = [_world(ctx, n) for n in (8, 22, 9)]
    streams = [torch.cuda.Stream() for _ in worlds]
    stop, rc = C.c_int(0), [None] * len(worlds)

    def run(k, each):
        w = worlds[k]
        rc[k] = loop(C.cast(w.lib.b3_stage_solve, C.c_void_p), C.cast(sync, C.c_void_p), w.h,
                     C.c_void_p(streams[k].cuda_stream), 4000, each, C.byref(stop))

    for each in (7, 8, 5, 6):
        threads = [threading.Thread(target=run, args=(k, each + k)) for k in range(len(worlds))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert rc == [0] * len(worlds), b3.load().b3_last_error()
    for w in worlds:
        assert w.counters()["timeouts"] == 0
        w.close()


def test_worlds_and_adjoints_on_two_threads(ctx):
    """Steps and gradients are those of the worlds alone, bit for bit."""
    import torch
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def make(k):
        w = scenes.build_world(ctx, [scenes.random_pile(51, n=40, hull_frac=0.0), scenes.c1(dims=(22, 22, 22))][k])
        return w, b3.Adjoint(w, 12, 3)

    def run(w, a, s):
        for _ in range(2):
            a.forward(stream=s)
            a.backward(d_pos=np.ones((w.n, 3), np.float32), stream=s)
            s.synchronize()
        return [*a.gradients().values(), *w.read_state(stream=s)]

    alone, both = [None, None], [None, None]
    for k in (0, 1):
        w, a = make(k)
        alone[k] = run(w, a, streams[k])
        a.close()
        w.close()
    made = [make(k) for k in (0, 1)]
    errors = []

    def guarded(k):
        try:
            both[k] = run(*made[k], streams[k])
        except Exception as e:  # noqa: BLE001 (handed to the main thread)
            errors.append(e)
    threads = [threading.Thread(target=guarded, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in (0, 1):
        for x, y in zip(alone[k], both[k]):
            assert np.array_equal(np.ascontiguousarray(x).view(np.uint32), np.ascontiguousarray(y).view(np.uint32))
        made[k][1].close()
        made[k][0].close()
