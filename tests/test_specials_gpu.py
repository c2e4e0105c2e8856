"""NaNs of both signs, infinities, zeros of both signs and denormals through the
one-CTA kernel, the cluster kernel, the threshold, the window and the pipeline: the
answers equal sorting by the order-preserving key."""
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


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [2, 1003, 16_000, 200_003, 700_001, 3_000_017])
@pytest.mark.parametrize("share", [0.0001, 0.2])
def test_specials(g, dtype, n, share):
    r = np.random.default_rng(n)
    x = r.standard_normal(n).astype(dtype)
    u = np.dtype(f"u{x.itemsize}").type
    sign = u(1 << (8 * x.itemsize - 1))
    nan = np.array([np.inf], dtype).view(u)[0]
    bits = np.concatenate([
        nan + u(1) + r.integers(0, 1000, 50).astype(u),        # NaNs, smallest payloads
        (nan + u(1) + r.integers(0, 1000, 50).astype(u)) | sign,
        np.array([~u(0), ~u(0) ^ sign, nan, nan | sign, u(0), sign, u(1), u(1) | sign], u)])
    count = max(2, int(n * share))
    x[r.integers(0, n, count)] = bits[r.integers(0, bits.size, count)].view(dtype)
    desc = key_sorted(x)[::-1]
    d = DeviceArray(x)
    edge = np.arange(1, min(n, 40) + 1)
    zero = int(np.count_nonzero(key_sorted(x)[::-1] > 0))  # (NaNs compare false)
    lists = [np.concatenate([edge, n + 1 - edge]), r.integers(1, n + 1, 101), [1], [n],
             [max(1, n // 2)], np.clip(np.arange(zero - 30, zero + 40, 7), 1, n),
             np.clip(np.arange(1, 900, 9), 1, n)]
    ctx = g.Context(0)
    for ks in lists:
        ks = np.array(ks, dtype=np.uint32)
        for small in (True, False):
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=small), desc[ks - 1],
                        f"{ks[:4]} small={small}")
    for K in sorted({1, min(n, 16), min(n, 1000), max(1, n // 64), max(1, n // 32)}):
        for pipeline in (False, True):
            assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx, pipeline=pipeline), desc[:K], f"top-{K}")
    ctx.close()
