"""The streaming passes' grid and bucket count at their steps: sizes around whole
CTAs' shares, one share per SM, and the sizes where the buckets double, through
the pipeline; and clustered k's on both sides of the size from which they leave
the one-launch path.  Every answer equals sorting."""
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


def values(dtype, n):
    r = np.random.default_rng(n)
    if dtype == np.uint32:
        return r.integers(0, 1 << 32, n, dtype=np.uint32)
    return r.standard_normal(n).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.uint32, np.float64])
@pytest.mark.parametrize("n", [1, 16384, 16385, 65535, 3 * 16384 - 1, 152 * 16384 - 1, 152 * 16384 + 1,
                               (1 << 22) + 1, (1 << 23) - 1, (1 << 24) + 3])
def test_pipeline_sizes(g, dtype, n):
    x = values(dtype, n)
    want = np.sort(x)[::-1]
    ks = np.unique(np.linspace(1, n, 333).astype(np.uint32))
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    got = g.multiselect_ptr(d.ptr, n, x.dtype, ks, ctx=ctx, small=False)
    assert_same(got, want[ks.astype(np.int64) - 1], f"n={n}")
    K = min(n, 5000)
    got = g.topk_ptr(d.ptr, n, x.dtype, K, ctx=ctx, pipeline=True)
    assert_same(got, want[:K], f"top-{K} of {n}")
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.uint32, np.float64])
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, 1 << 20])
def test_clustered_ks(g, dtype, n):
    x = values(dtype, n)
    want = np.sort(x)[::-1]
    d = DeviceArray(x)
    for ks in ([n // 2], [1], [n], np.arange(n // 3, n // 3 + 900), [n // 2, n // 2 + n // 32 - 1],
               [n // 2, n // 2 + n // 32]):
        ks = np.asarray(ks, dtype=np.uint32)
        got = g.multiselect_ptr(d.ptr, n, x.dtype, ks)
        assert_same(got, want[ks.astype(np.int64) - 1], f"n={n} k={ks[0]}")
    one = x.copy()
    one[:] = x[0]
    d = DeviceArray(one)
    got = g.multiselect_ptr(d.ptr, n, x.dtype, np.array([n // 2], np.uint32))
    assert_same(got, one[:1], "one value")
