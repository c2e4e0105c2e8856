"""Around the numbers of requests at which a vector's table gets fewer buckets: every
answer equals sorting, for k lists and for the same number of largest values."""
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
@pytest.mark.parametrize("n", [(1 << 23) + 5, (1 << 24) + 3])
def test_many(g, dtype, n):
    r = np.random.default_rng(n)
    x = (r.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) if dtype == np.uint32
         else r.standard_normal(n).astype(dtype))
    desc = np.sort(x)[::-1]
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    for count in (8192, 16383, 16384, 32767, 32768, 70_001):
        ks = r.integers(1, n + 1, count).astype(np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx), desc[ks - 1], f"{count} k's")
    assert_same(g.topk_ptr(d.ptr, n, dtype, 40_000, ctx=ctx, pipeline=True), desc[:40_000], "top-k")
    ctx.close()
