"""Radix sort at the sizes where it takes other paths: around the one-block
sort's capacities, around a key per thread of the whole grid, and ranges that
end inside a tile; key widths of one to four passes; keys, pairs and records;
on a side stream and inside a CUDA graph."""
import numpy as np
import pytest
import torch

from experiments_b200 import b3

pytestmark = pytest.mark.gpu

GRID = 148 * 1024
SIZES = [31, 1024, 1025, 4097, 8191, 8192, 8193, GRID - 1, GRID + 1, 2 * GRID + 77, 4 * GRID + 1, 8 * GRID + 4097]


def _keys(n, bits, dist, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if dist == "skewed":  # most keys equal, the rest anywhere
        k[rng.random(n) < 0.95] = np.uint32((1 << bits) - 1)
    return k


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits,dist", [(1, "even"), (9, "even"), (17, "skewed"), (32, "even")])
def test_sizes(ctx, n, bits, dist):
    keys = _keys(n, bits, dist, n + bits)
    order = np.argsort(keys, kind="stable")
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    dv = torch.arange(n, device="cuda", dtype=torch.int32)
    sort = b3.RadixSort32(ctx)
    ko, vo = torch.empty_like(dk), torch.empty_like(dv)
    sort.execute_out(dk, ko, dv, vo, key_bits=bits)
    rec = torch.stack([dk, dv], 1).contiguous()
    sort.execute_sortdata(rec, key_bits=bits)
    only = dk.clone()
    sort.execute(only, key_bits=bits)
    torch.cuda.synchronize()
    want_k, want_v = keys[order].view(np.int32), order.astype(np.int32)
    assert np.array_equal(ko.cpu().numpy(), want_k) and np.array_equal(vo.cpu().numpy(), want_v)
    assert np.array_equal(rec.cpu().numpy(), np.stack([want_k, want_v], 1))
    assert np.array_equal(only.cpu().numpy(), want_k)
    assert np.array_equal(dk.cpu().numpy(), keys.view(np.int32))  # out of place: the input is only read


@pytest.mark.parametrize("n", [5000, 200001])
def test_in_a_graph_and_on_a_stream(ctx, n):
    sort = b3.RadixSort32(ctx)
    src = torch.from_numpy(_keys(n, 24, "even", 3).view(np.int32)).cuda()
    buf, vals = src.clone(), torch.arange(n, device="cuda", dtype=torch.int32)
    iota = vals.clone()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        sort.execute(buf, vals, key_bits=24, stream=st)  # grows the scratch before the capture
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        buf.copy_(src)
        vals.copy_(iota)
        sort.execute(buf, vals, key_bits=24, stream=st)
    for seed in (4, 5):
        keys = _keys(n, 24, "even", seed)
        src.copy_(torch.from_numpy(keys.view(np.int32)))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(buf.cpu().numpy().view(np.uint32), keys[order])
        assert np.array_equal(vals.cpu().numpy(), order.astype(np.int32))


@pytest.mark.parametrize("n", [0, 1, 4096, 4097, 40 * 4096 + 5, 3000001])
def test_scan_totals(ctx, n):
    """The scan's look-back takes 32 tiles at a time: below, at and past that."""
    rng = np.random.default_rng(n)
    a = rng.integers(0, 5, max(n, 1)).astype(np.int32)[:n]
    src = torch.from_numpy(a).cuda() if n else torch.zeros(1, device="cuda", dtype=torch.int32)
    dst = torch.empty_like(src)
    total = b3.PrefixScan(ctx).execute(src, dst, n=n)
    assert total == int(a.sum())
    if n:
        assert np.array_equal(dst.cpu().numpy(), np.concatenate([[0], np.cumsum(a)[:-1]]).astype(np.int32))
