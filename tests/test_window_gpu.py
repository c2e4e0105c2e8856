"""Clustered ranks through the sampled window (csrc/ggks_window.cuh): one k, k's
close together and long top-k's, of vectors around the path's smallest size and
ragged ones, in every type; windows open at either end; bins that hold many
copies of one key, the keys beyond the sampled extremes, and both kinds of miss
(a sample that misrepresents the vector, a large bin of distinct keys), which
the pipeline answers.  Every answer equals sorting by the order-preserving
key."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same
from test_spec_gpu import sampled_positions

pytestmark = pytest.mark.gpu

MIN_N = 1 << 18  # the path takes larger vectors


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


def key_sorted(x):
    if x.dtype == np.uint32:
        return np.sort(x)
    u = np.dtype(f"u{x.itemsize}").type
    b, top = x.view(u), u(1 << (8 * x.itemsize - 1))
    return x[np.argsort(np.where(b & top, ~b, b | top), kind="stable")]


def make(dtype, dist, n):
    r = np.random.default_rng(n)
    if dist == "ints":
        x = r.integers(0, 200, n) * (r.random(n) < 0.6)  # 40 % zeros and more
    elif dist == "sorted":
        x = np.sort(r.standard_normal(n) * 1e5 + 1e6)
    elif dist == "heavy":
        x = np.abs(r.standard_cauchy(n))
    else:
        x = r.random(n) * 1e9
    return np.minimum(x, 4e9).astype(dtype)


def run(g, fn, *args, **kw):
    ctx = g.Context(0)
    try:
        got = fn(*args, ctx=ctx, small=False, **kw)
        return got, ctx.stats()
    finally:
        ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("dist", ["spread", "heavy", "ints", "sorted"])
@pytest.mark.parametrize("n", [MIN_N + 1, 1_000_003])
def test_window(g, dtype, dist, n):
    x = make(dtype, dist, n)
    desc = key_sorted(x)[::-1]
    d = DeviceArray(x, pad_front=n % 3)
    lists = [[n // 2], [1], [n], [n // 3, n // 3 + 7, n // 3], list(range(1, 1025)),
             list(range(n - 700, n + 1)), list(range(n // 7, n // 7 + n // 32, n // 32000 + 1))[:1024]]
    for ks in lists:
        ks = np.array(ks, dtype=np.uint32)
        got, st = run(g, g.multiselect_ptr, d.ptr, n, dtype, ks)
        assert_same(got, desc[ks - 1], f"{dist} {n} {ks[:3]}")
        # (few-valued vectors may hold more copies around a k than are kept)
        few = dist == "ints" or (dist == "heavy" and dtype == np.uint32)
        assert st["spec_calls"] == 1 or few
    for K in (4097, 5000, n // 32):
        got, st = run(g, g.topk_ptr, d.ptr, n, dtype, K)
        assert_same(got, desc[:K], f"{dist} {n} top-{K}")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_window_misses(g, dtype):
    """The largest elements are never sampled (the window's keys fall short or the
    end bin holds thousands of distinct keys); a cluster of distinct keys far
    narrower than a bin."""
    n = 1 << 20
    r = np.random.default_rng(5)
    x = r.random(n)
    free = np.setdiff1d(np.arange(n), np.unique(sampled_positions(n).astype(np.int64)))
    x[r.choice(free, 6000, replace=False)] = 2.0 + r.random(6000)
    y = r.random(n)
    y[r.choice(n, 20000, replace=False)] = 1.0 + np.arange(20000) * (2.0 ** -22 if dtype == np.float32 else 2.0 ** -50)
    y[r.choice(n, 50, replace=False)] = 1e30
    for v in (x, y):
        v = v.astype(dtype)
        desc = key_sorted(v)[::-1]
        d = DeviceArray(v)
        for K in (5000, 9000):
            got, _ = run(g, g.topk_ptr, d.ptr, n, dtype, K)
            assert_same(got, desc[:K], f"top-{K}")
        for ks in ([3000], [10000], [n // 2]):
            ks = np.array(ks, dtype=np.uint32)
            got, _ = run(g, g.multiselect_ptr, d.ptr, n, dtype, ks)
            assert_same(got, desc[ks - 1], str(ks))


def test_window_host_vectors_and_device_output(g):
    import torch
    n = 700_001
    x = make(np.float32, "spread", n)
    desc = np.sort(x)[::-1]
    pinned = torch.empty(n, dtype=torch.float32, pin_memory=True)
    pinned.numpy()[:] = x
    for v in (x, pinned.numpy()):
        assert_same(g.multiselect_host(v, np.array([n // 2], np.uint32)), desc[[n // 2 - 1]], "host")
        assert_same(g.topk_host(v, 9000), desc[:9000], "host top-k")
    d = DeviceArray(x)
    out = torch.zeros(9001, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g.topk_ptr(d.ptr, n, np.float32, 9000, out_device_ptr=out.data_ptr())
    assert_same(out.cpu().numpy()[:9000], desc[:9000], "device output")
    assert out[9000].item() == 0
