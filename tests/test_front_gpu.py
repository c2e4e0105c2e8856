"""The sampling kernels and the plan of up to 1024 sorted requests
(csrc/ggks_front.cuh, k_plan_few) where they can go wrong: vectors around the
sample's size and its CTAs', request counts around a sorting CTA's share and the
plan's limit, repeated and unsorted k's, spans of a few keys, one key and one
far outlier; and thresholds whose fine slice holds more samples than are ranked.
Every answer equals sorting."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same

pytestmark = pytest.mark.gpu

SIZES = [100, 1023, 2047, 8193, 65535, 65536, 65537, 131_073]
COUNTS = [1, 31, 32, 33, 64, 65, 1000, 1023, 1024, 1025]


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


def make(dtype, dist, n):
    r = np.random.default_rng(n)
    if dist == "spread":
        x = r.random(n) * 1e6
    elif dist == "sorted":
        x = np.sort(r.random(n)) * 1e6
    elif dist == "few":
        x = 1.0 + r.integers(0, 3, n)
    else:  # one key and an outlier
        x = np.full(n, 7.0)
        x[n // 2] = 4e9
    return x.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("dist", ["spread", "sorted", "few", "outlier"])
def test_requests_and_sizes(g, dtype, dist):
    ctx = g.Context(0)
    for i, n in enumerate(SIZES):
        x = make(dtype, dist, n)
        want = np.sort(x)[::-1]
        d = DeviceArray(x, pad_front=i % 3)
        r = np.random.default_rng(n)
        for count in COUNTS[i % 2::2]:
            ks = r.integers(1, n + 1, count).astype(np.uint32)
            ks[::3] = ks[0]
            ks[-1] = n
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=False), want[ks - 1],
                        f"{dist} n={n} {count} k's")
    ctx.close()


@pytest.mark.parametrize("values", [2, 40, 3000, 1 << 30])
def test_threshold_slices(g, values):
    """65536 samples over `values` distinct keys: a fine slice holds from a few
    samples to all of them."""
    n = 1 << 21
    x = np.random.default_rng(values).integers(0, values, n).astype(np.uint32)
    want = np.sort(x)[::-1]
    d = DeviceArray(x)
    for K in (1, 100, 4096):
        assert_same(g.topk_ptr(d.ptr, n, np.uint32, K), want[:K], f"top-{K} of {values} values")
