"""Segments of the cluster kernel by their size: hundreds of requested buckets of a few
keys in one CTA (a top-k of distinct doubles), segments around one vote, and
segments of copies of one key, in every type."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("kind", ["distinct", "runs", "copies", "mixed"])
@pytest.mark.parametrize("n", [33_001, 120_007, 250_003])
def test_segments(g, dtype, kind, n):
    r = np.random.default_rng(n)
    if kind == "distinct":
        x = r.permutation(n) * 977.0
    elif kind == "runs":  # 1 to 70 copies of each value
        x = np.repeat(r.permutation(n), r.integers(1, 71, n))[:n] * 3.0
    elif kind == "copies":
        x = r.integers(0, 256, n) * 1.0
    else:
        x = np.where(r.random(n) < 0.5, r.integers(0, 200, n) * 1000.0, r.random(n) * 2e5)
    x = r.permutation(x).astype(dtype)
    desc = np.sort(x)[::-1]
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    for K in (1, 33, 900, 1024):
        assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx), desc[:K], f"top-{K}")
    for ks in (r.integers(1, n + 1, 1024), np.arange(n // 3, n // 3 + 1000), np.repeat(r.integers(1, n + 1, 200), 5)):
        ks = ks.astype(np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx), desc[ks - 1])
    st = ctx.stats()
    ctx.close()
    assert st["small_calls"] + st["small_misses"] == 7
