"""Sweep-and-prune pair kernel where its warps and tiles end: remainders of 32
proxies, sweeps that stop inside a tile, more partners than the counting pass
keeps, each axis, unsorted records and a capacity below the count, against the
oracle's pairs in order."""
import numpy as np
import pytest

import oracle
from experiments_b200 import b3, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sap():
    c = b3.Context(0)
    yield b3.SapPairs(c)
    c.close()


def _records(n, span, seed, special=False):
    lo = scenes.uniform(seed, 1, 3 * n, 0.0, span).reshape(n, 3).astype(np.float32)
    hi = lo + scenes.uniform(seed, 2, 3 * n, 0.2, 1.5).reshape(n, 3).astype(np.float32)
    if special:
        hi[::7, 0] = np.inf
        lo[3::11, 1] = -np.inf
        hi[5::13, 2] = lo[5::13, 2] - 1.0
    rec = np.zeros((n, 8), np.float32)
    rec[:, 0:3], rec[:, 4:7] = lo, hi
    ids = scenes.uniform(seed, 3, n, 0.0, 1.0).argsort().astype(np.int32)
    rec[:, 3], rec[:, 7] = ids.view(np.float32), ids.view(np.float32)
    return rec


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n,span", [(1, 1.0), (2, 1.0), (31, 3.0), (32, 1.0), (33, 3.0), (64, 20.0), (65, 2.0), (700, 4.0),
                                    (5000, 30.0)])
def test_pairs_in_order(sap, n, span, axis, special):
    import torch
    rec = _records(n, span, 31 + n, special)
    for order in (rec[:, axis].argsort(kind="stable"), np.arange(n)):
        s = np.ascontiguousarray(rec[order])
        exp = oracle.sap_sorted_pairs(s, axis)
        for cap in (len(exp) + 3, len(exp) // 2 + 1):
            d_p = torch.full((cap, 2), -1, dtype=torch.int32, device="cuda")
            d_c = torch.zeros(1, dtype=torch.int32, device="cuda")
            sap.execute(torch.from_numpy(s).cuda(), d_p, d_c, axis=axis, max_pairs=cap)
            k = min(cap, len(exp))
            assert int(d_c.item()) == len(exp)
            got = d_p.cpu().numpy()
            assert np.array_equal(got[:k], exp[:k]) and (got[k:] == -1).all()


@pytest.mark.parametrize("statics", [1, 40])
def test_static_bodies_come_first(statics):
    """Worlds with few and many static bodies against the oracle's pair list."""
    from helpers import make_pair
    c = b3.Context(0)
    n = 300
    pos = np.concatenate([np.stack([np.arange(statics) * 1.1, np.full(statics, 0.2), np.full(statics, 3.0)], 1),
                          scenes.uniform(5, 1, 3 * n, 0.0, 6.0).reshape(n, 3)])
    m = statics + n
    b = scenes._bodies(np.zeros(m, np.int32), np.concatenate([np.zeros(statics), np.ones(n)]), pos,
                       np.tile([0.0, 0.0, 0.0, 1.0], (m, 1)), np.full(m, 0.5), np.zeros(m))
    sc = scenes.Scene(name="statics", shapes=[scenes.box_vertices(0.5, 0.5, 0.5)], num_worlds=1, config={}, **b)
    w, o = make_pair(c, sc, flags=b3.B3_WORLD_SAP_BROADPHASE)
    for x in (w, o):
        x.stage("aabbs")
        x.stage("broadphase")
    assert len(o.pairs()) > 0 and np.array_equal(w.pairs(), o.pairs())
    w.close()
    o.close()
    c.close()
