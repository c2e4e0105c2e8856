"""Clustered ranks and top-k's of vectors in which a few values make up most of the
elements: the copies of a popular window end or threshold are counted, not kept.
Ranks on both sides of every boundary between values; -inf, +inf and NaNs of both
signs among the values; the answers equal sorting by the order-preserving key
and none needs the pipeline."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same
from test_window_gpu import key_sorted

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


def values(dtype, kind):
    if kind == "special":
        if dtype == np.uint32:
            return np.array([0, 1, 0x7FFFFFFF, 0x80000000, 0xFFFFFFFE, 0xFFFFFFFF], dtype)
        u = np.dtype(f"u{np.dtype(dtype).itemsize}").type
        nan = np.array([np.inf], dtype).view(u)[0] + u(1)
        sign = u(1 << (8 * np.dtype(dtype).itemsize - 1))
        bits = np.array([nan, nan | sign, ~u(0), ~u(0) >> u(1)], u).view(dtype)
        return np.concatenate([bits, np.array([-np.inf, -1, -0.0, 0.0, 1e-30, np.inf], dtype)])
    return (np.arange(kind) + 1).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("kind", [1, 2, 10, "special"])
@pytest.mark.parametrize("others", [0, 0.3])
def test_popular(g, dtype, kind, others):
    n = 3_000_017
    r = np.random.default_rng(7)
    vals = values(dtype, kind)
    x = vals[r.integers(0, vals.size, n)]
    if others:  # and distinct values between and around them
        at = r.random(n) < others
        x[at] = (r.random(np.count_nonzero(at)) * 12).astype(dtype)
    desc = key_sorted(x)[::-1]
    step = np.flatnonzero(desc[1:].view(f"u{x.itemsize}") != desc[:-1].view(f"u{x.itemsize}")) + 1
    edges = step if step.size < 40 else step[r.integers(0, step.size, 12)]
    for p in (n // 5, n // 2):  # where a popular value begins
        edges = np.append(edges, step[np.argmin(np.abs(step - p))] if step.size else p)
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    for e in edges:
        for ks in ([e], [e + 1], [max(1, e - 300), e, min(n, e + 1), min(n, e + 2000)]):
            ks = np.array(ks, dtype=np.uint32).clip(1, n)
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=False), desc[ks - 1],
                        f"{kind} {ks}")
    for K in (1, 16, 1000, 4096, 4097, 20000, n // 32):
        assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx), desc[:K], f"{kind} top-{K}")
    if not others:
        assert ctx.stats()["topk_misses"] == 0
    ctx.close()


def test_popular_host_vector(g):
    """The pass also writes the device copy, here of a vector that most of its keys
    are not kept from."""
    import torch
    n = 1_000_003
    x = (np.random.default_rng(1).integers(0, 3, n) * 2).astype(np.float32)
    desc = np.sort(x)[::-1]
    pinned = torch.empty(n, dtype=torch.float32, pin_memory=True)
    pinned.numpy()[:] = x
    for k in (1, n // 3, n // 3 + 500, n // 2, n):
        got = g.multiselect_host(pinned.numpy(), np.array([k], np.uint32))
        assert_same(got, desc[[k - 1]], str(k))
    for K in (1000, 5000):
        assert_same(g.topk_host(pinned.numpy(), K), desc[:K], f"top-{K}")
