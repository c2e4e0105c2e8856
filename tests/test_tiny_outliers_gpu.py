"""Tiny vectors whose keys crowd into few of the bins because some values lie far
out: bins just below and above what a warp sorts, and most of the vector in one bin,
answered by the one-CTA kernel."""
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


@pytest.mark.parametrize("far", [np.inf, 1e30, -1e30])
@pytest.mark.parametrize("n", [16_384, 24_000, 32_768])
def test_far_out(g, far, n):
    r = np.random.default_rng(n)
    x = r.random(n).astype(np.float32)
    x[r.integers(0, n, 20)] = far
    desc = np.sort(x)[::-1]
    d = DeviceArray(x)
    ctx = g.Context(0)
    for ks in (r.integers(1, n + 1, 1000), np.arange(1, 60), np.linspace(1, n, 101).astype(int)):
        ks = ks.astype(np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, np.float32, ks, ctx=ctx), desc[ks - 1])
    st = ctx.stats()
    ctx.close()
    assert st["small_calls"] == 3 and st["launches"] == 3  # (a miss launches the next kernel)


@pytest.mark.parametrize("crowd", [255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1500])
def test_one_bin(g, crowd):
    """A bin of `crowd` distinct keys (2^18 keys wide here), among spread ones."""
    r = np.random.default_rng(crowd)
    x = r.integers(0, 1 << 31, 5000).astype(np.uint32)
    x[:2] = [0, (1 << 31) - 1]
    x = x[(x >> 18) != 77]
    x = r.permutation(np.append(x, (77 << 18) + r.choice(1 << 18, crowd, replace=False)).astype(np.uint32))
    desc = np.sort(x)[::-1]
    ks = np.arange(1, x.size + 1, 6).astype(np.uint32)
    d = DeviceArray(x)
    got = g.multiselect_ptr(d.ptr, x.size, np.uint32, ks)
    assert_same(got, desc[ks - 1])


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("n", [40, 616, 5563, 16_384, 32_768])
def test_crowd(g, dtype, n):
    """Nine tenths of the vector within a sliver of its range, in one bin or two."""
    if n > 16_384 and dtype == np.float64:
        n = 16_384
    r = np.random.default_rng(n)
    x = (1e6 + r.random(n) * 30_000).astype(dtype) if dtype == np.uint32 else (1000 + r.random(n) * 0.05).astype(dtype)
    at = r.random(n) < 0.1
    x[at] = (r.random(np.count_nonzero(at)) * (4e9 if dtype == np.uint32 else 1e30)).astype(dtype)
    desc = np.sort(x)[::-1]
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    for ks in (r.integers(1, n + 1, 1000), [1], [n], [n // 2], np.linspace(1, n, 30).astype(int)):
        ks = np.array(ks, dtype=np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx), desc[ks - 1])
    assert_same(g.topk_ptr(d.ptr, n, dtype, min(n, 1024), ctx=ctx), desc[:1024])
    st = ctx.stats()
    ctx.close()
    assert st["small_calls"] == 6 and st["launches"] == 6
