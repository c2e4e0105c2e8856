"""Window attempts that miss are counted, and a vector that the one-launch path takes
goes to it after a miss, not to the pipeline."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same
from test_spec_gpu import sampled_positions

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
@pytest.mark.parametrize("n,small", [(1 << 20, True), (1 << 20, False), ((1 << 20) + 1, True)])
def test_miss(g, dtype, n, small):
    """The largest elements are never sampled, so the window lies too low."""
    r = np.random.default_rng(5)
    x = r.random(n).astype(dtype)
    free = np.setdiff1d(np.arange(n), np.unique(sampled_positions(n).astype(np.int64)))
    x[r.choice(free, 9000, replace=False)] = 2.0 + r.random(9000).astype(dtype)
    ks = np.array([12000, 12500], dtype=np.uint32)
    d = DeviceArray(x)
    ctx = g.Context(0)
    got = g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=small)
    st = ctx.stats()
    ctx.close()
    assert_same(got, np.sort(x)[::-1][ks - 1])
    assert st["topk_misses"] == 1
    assert st["small_calls"] == (1 if small and n <= 1 << 20 else 0)
