"""Windows whose candidates crowd into a few of the equal-width bins: a gap in the key
range (two modes, values far out), values with many copies.  A large bin of one
key is answered as it is; a large bin of distinct keys is selected from again, on
its keys alone.  Every answer equals sorting and none needs the pipeline."""
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
@pytest.mark.parametrize("device_out", [False, True])
def test_gap(g, dtype, device_out):
    import torch
    n = 10_000_019
    r = np.random.default_rng(11)
    if dtype == np.uint32:
        x = (r.integers(0, 1 << 22, n) + (r.random(n) < 0.5) * 4_000_000_000).astype(dtype)
    else:
        x = ((1 + r.random(n)) * r.choice([-1, 1], n)).astype(dtype)
    desc = np.sort(x)[::-1]
    mid = int(np.count_nonzero(x > (0 if dtype != np.uint32 else 1 << 31)))
    d = DeviceArray(x, pad_front=1)
    ctx = g.Context(0)
    out = torch.zeros(16, dtype={4: torch.int32, 8: torch.int64}[x.itemsize], device="cuda")
    torch.cuda.synchronize()
    for ks in ([mid], [mid + 1], [mid + 4000, mid - 4000, mid + 1, mid, mid - 4000, mid + 5]):
        ks = np.array(ks, dtype=np.uint32)
        if device_out:
            g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, out_device_ptr=out.data_ptr())
            got = out.cpu().numpy()[:ks.size].view(dtype)
        else:
            got = g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx)
        assert_same(got, desc[ks - 1], str(ks))
    st = ctx.stats()
    assert st["topk_misses"] == 0 and 3 <= st["recursions"] <= 4  # a bin's requests together
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
def test_copies(g, dtype):
    """256 values: 78 thousand copies of each, more than a CTA selects from."""
    n = 20_000_003
    r = np.random.default_rng(12)
    x = r.integers(0, 256, n).astype(dtype)
    desc = np.sort(x)[::-1]
    d = DeviceArray(x)
    ctx = g.Context(0)
    for at in (0.2, 0.5, 0.77):
        k = int(n * at)
        for ks in ([k], list(range(k, k + n // 40, n // 400))):
            ks = np.array(ks, dtype=np.uint32)
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx), desc[ks - 1], str(ks[:2]))
    for K in (5000, 100_000):
        assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx), desc[:K], f"top-{K}")
    st = ctx.stats()
    assert st["topk_misses"] == 0 and st["recursions"] == 0
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("far", [300, 7000])
def test_topk_over_a_gap(g, dtype, far):
    """A top-k of values far out (distinct ones, or copies of one) and of the crowd below them."""
    n = 4_000_037
    r = np.random.default_rng(13)
    for same in (True, False):
        x = r.random(n)
        x[r.choice(n, far, replace=False)] = 1e30 if same else 1e30 * (1 + r.random(far))
        x = x.astype(dtype)
        desc = np.sort(x)[::-1]
        d = DeviceArray(x)
        ctx = g.Context(0)
        for K in (far, far + 1, 20_000, 60_000):
            assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx), desc[:K], f"{same} top-{K}")
        ks = np.array([far, far + 1, far + 9000], dtype=np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx), desc[ks - 1], str(ks))
        ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dist", ["normal", "cauchy"])
def test_topk_tail(g, dtype, dist):
    """The few hundred keys past the sample's largest spread over the open end's bins."""
    n = 40_000_003
    r = np.random.default_rng(14)
    x = (100 + r.standard_normal(n) if dist == "normal" else r.standard_cauchy(n)).astype(dtype)
    top = np.sort(np.partition(x, n - 30_000)[-30_000:])[::-1]
    d = DeviceArray(x)
    ctx = g.Context(0)
    for K in (4500, 9000, 20_000, 30_000):
        assert_same(g.topk_ptr(d.ptr, n, dtype, K, ctx=ctx), top[:K], f"{dist} top-{K}")
    st = ctx.stats()
    assert st["topk_misses"] == 0 and st["recursions"] == 0
    ctx.close()
