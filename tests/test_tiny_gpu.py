"""One-CTA selection of tiny vectors (csrc/ggks_tiny.cuh): sizes around a warp, a
CTA and the largest vector it takes (32768 elements of 4 bytes, 16384 of 8),
values that crowd into few bins (one key, two keys, both signs around the
exponent gap, far outliers, tight clusters that it leaves to the cluster
kernel), every rank or few, and top-k.  Every answer equals sorting by the
order-preserving key."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 1000, 1024, 1025, 8191, 16383, 16384, 16385, 32767, 32768, 32769]


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
    if dtype == np.uint32:
        return {"spread": r.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32),
                "crowd": (7 + 3000 * (r.random(n) < 0.5)).astype(np.uint32),
                "edge": np.where(r.random(n) < 0.5, 0, 0xFFFFFFFF).astype(np.uint32)}[dist]
    if dist == "spread":
        return r.standard_normal(n).astype(dtype)
    if dist == "crowd":  # a tight cluster, copies of it, and far outliers
        x = (1.0 + r.integers(0, 1 << 12, n) * np.finfo(dtype).eps).astype(dtype)
        x[r.random(n) < 0.3] = 1.5
        x[0], x[-1] = -3e38, 3e38
        return x
    x = r.standard_normal(n).astype(dtype)
    x[::3] = 0.0
    x[1::3] = -0.0
    x[2::7] = np.inf
    x[5::11] = -np.inf
    return x


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("dist", ["spread", "crowd", "edge"])
def test_tiny(g, dtype, dist):
    ctx = g.Context(0)
    for n in SIZES:
        x = make(dtype, dist, n)
        want = key_sorted(x)
        d = DeviceArray(x, pad_front=n % 3)
        for count in {1, min(n, 11), min(n, 1024)}:
            ks = np.unique(np.linspace(1, n, count).astype(np.uint32))
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx),
                        want[n - ks.astype(np.int64)], f"{dist} n={n} {count} k's")
            assert_same(g.topk_ptr(d.ptr, n, dtype, count, ctx=ctx), want[::-1][:count],
                        f"{dist} n={n} top-{count}")
    ctx.close()
