"""The splitter table of 8-byte keys (2^12 slices in four copies; up to 2^10 per
problem of a batch) where a slice can go wrong: a span that covers both signs
and every exponent, a span of a few ulps, denormals and infinities, and sizes
around the sample's.  Every answer equals sorting by the order-preserving key
(-0.0 below +0.0)."""
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


def make(dist, n):
    r = np.random.default_rng(n)
    if dist == "pm1e6":
        return r.uniform(-1e6, 1e6, n)
    if dist == "every_exponent":
        return np.ldexp(r.uniform(-1.0, 1.0, n), r.integers(-1074, 1024, n))
    if dist == "few_ulps":
        return 1.0 + r.integers(0, 5000, n) * 2.0 ** -52
    x = np.ldexp(r.integers(-1000, 1000, n).astype(np.float64), -1074)  # denormals
    x[r.integers(0, n, 50)] = np.inf
    x[r.integers(0, n, 50)] = -np.inf
    return x


def key_sorted(x):
    b = x.view(np.uint64)
    key = np.where(b >> np.uint64(63), ~b, b | np.uint64(1 << 63))
    return x[np.argsort(key, kind="stable")]


@pytest.mark.parametrize("dist", ["pm1e6", "every_exponent", "few_ulps", "denormals"])
@pytest.mark.parametrize("n", [4097, 65537, (1 << 21) + 3])
def test_f64_table(g, dist, n):
    x = make(dist, n)
    want = key_sorted(x)
    ks = np.unique(np.linspace(1, n, 700).astype(np.uint32))
    d = DeviceArray(x)
    for small in (True, False):
        ctx = g.Context(0)
        got = g.multiselect_ptr(d.ptr, n, x.dtype, ks, ctx=ctx, small=small)
        assert_same(got, want[n - ks.astype(np.int64)], f"{dist} {n} small={small}")
        if dist == "pm1e6" and n > 1 << 20:
            # 700 buckets of 8192, none much fuller than the others
            assert ctx.stats()["survivors"] < 2 * 700 * n / 8192
        ctx.close()
    got = g.multiselect_batch_ptr([d.ptr, d.ptr], [n, n // 2], x.dtype, [ks, ks[:100]])
    assert_same(got[0], want[n - ks.astype(np.int64)], f"batch {dist} {n}")
    half = key_sorted(x[:n // 2])
    assert_same(got[1], half[n // 2 - ks[:100].astype(np.int64)], f"batch {dist} {n // 2}")
