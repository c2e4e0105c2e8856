"""A batch's tiles are placed by length class: problems whose lengths sit at the
edges of a tile (whole tiles only, one element more, one less), many classes at
once, problems without requests between them, and requests that speculate (a
single k, a short top-k) next to ones that do not.  Every answer equals sorting."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 63, 64, 65, 65535, 65536, 65537, 2 * 65536, 3 * 65536 - 1, (1 << 18) - 1, 1 << 18,
         (1 << 18) + 1, (1 << 19) + 255, 3 << 18, (1 << 20) + 17]


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


@pytest.mark.parametrize("dtype", [np.float32, np.uint32, np.float64])
@pytest.mark.parametrize("copies", [1, 12])
def test_batch_tiles(g, dtype, copies):
    r = np.random.default_rng(copies)
    lens = EDGES * copies
    r.shuffle(lens)
    x = (r.integers(0, 1 << 32, max(lens), dtype=np.uint32).astype(dtype)
         if dtype == np.uint32 else r.standard_normal(max(lens)).astype(dtype))
    want = {n: np.sort(x[:n])[::-1] for n in set(lens)}
    d = DeviceArray(x)
    ks = []
    for i, n in enumerate(lens):
        m = (0, 1, 2, min(n, 40))[i % 4]
        k = np.unique(r.integers(1, n + 1, m))
        ks.append(r.permutation(k).astype(np.uint32))  # any order
    got = g.multiselect_batch_ptr([d.ptr] * len(lens), lens, x.dtype, ks)
    for n, k, o in zip(lens, ks, got):
        assert_same(o, want[n][k.astype(np.int64) - 1], f"n={n} k={k[:4]}")
    Ks = [min(n, 1 + 7 * (i % 9)) for i, n in enumerate(lens)]
    got = g.topk_batch_ptr([d.ptr] * len(lens), lens, x.dtype, Ks)
    for n, k, o in zip(lens, Ks, got):
        assert_same(o, want[n][:k], f"top {k} of {n}")


@pytest.mark.parametrize("bad", [0, 5001, 0xFFFFFFFF])
def test_batch_k_out_of_range(g, bad):
    d = DeviceArray(np.arange(5000, dtype=np.float32))
    ks = np.arange(1, 41, dtype=np.uint32)
    ks[17] = bad
    with pytest.raises(Exception):
        g.multiselect_batch_ptr([d.ptr, d.ptr], [5000, 5000], np.float32, [ks[:3], ks])


@pytest.mark.parametrize("dtype", [np.float32, np.uint32, np.float64])
@pytest.mark.parametrize("values", ["many", "few", "sorted"])
def test_batch_totals(g, dtype, values):
    """Problems of 1, 2, 8, 9 and 17 tiles: bucket totals come from the rows of up
    to eight tiles and by atomics beyond, a problem's only tile takes whole
    segments, and more than 512 slots leave a thread more than one."""
    tile = 65536
    r = np.random.default_rng(5)
    lens = [100, tile - 3, tile, tile + 1, 8 * tile, 8 * tile + 1, 17 * tile - 9]
    x = r.integers(0, 50 if values == "few" else 1 << 32, max(lens), dtype=np.uint32)
    x = x.astype(dtype) if dtype == np.uint32 or values == "few" else \
        r.standard_normal(max(lens)).astype(dtype)
    if values == "sorted":
        x = np.sort(x)
    d = DeviceArray(x)
    ctx = g.Context(0)
    g.batch_set_tuning(ctx, 16, tile)
    ks = [np.unique(r.integers(1, n + 1, 1500)).astype(np.uint32) for n in lens]
    got = g.multiselect_batch_ptr([d.ptr] * len(lens), lens, x.dtype, ks, ctx=ctx)
    for n, k, o in zip(lens, ks, got):
        assert_same(o, np.sort(x[:n])[::-1][k.astype(np.int64) - 1], f"n={n}")
    ctx.close()
