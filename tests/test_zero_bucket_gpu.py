"""Segments whose keys crowd into a corner of their bucket's key range (the bucket
around zero of zero-centred doubles spans every exponent): a segment that fits a
finishing CTA's buffer is sorted there, in a single call and in a batch, and no
recursive level runs for it."""
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


def around_zero(x, r, spread):
    """k's of the 400 elements nearest zero, and others over the whole vector."""
    n, mid = x.size, int(np.count_nonzero(x > 0))
    near = np.arange(mid - 200, mid + 200, 3)
    return np.concatenate([near, r.integers(1, n + 1, spread)]).astype(np.uint32)


@pytest.mark.parametrize("n,spread", [(3_000_017, 1500), (1 << 24, 60_000)])
def test_single(g, n, spread):
    r = np.random.default_rng(n)
    x = r.standard_normal(n)
    ks = around_zero(x, r, spread)
    d = DeviceArray(x)
    ctx = g.Context(0)
    got = g.multiselect_ptr(d.ptr, n, x.dtype, ks, ctx=ctx)
    st = ctx.stats()
    ctx.close()
    assert_same(got, np.sort(x)[::-1][ks - 1])
    assert st["recursions"] == 0


def test_batch(g):
    r = np.random.default_rng(3)
    vecs = [r.standard_normal(n) for n in (70_001, 300_007, 1_000_003, 2_000_003)]
    ks = [around_zero(x, r, 100) for x in vecs]
    bufs = [DeviceArray(x) for x in vecs]
    ctx = g.Context(0)
    got = g.multiselect_batch_ptr([b.ptr for b in bufs], [x.size for x in vecs], np.float64, ks, ctx=ctx)
    st = ctx.stats()
    ctx.close()
    for x, k, o in zip(vecs, ks, got):
        assert_same(o, np.sort(x)[::-1][k - 1])
    assert st["recursions"] == 0
