"""One k and clustered k's in the middle of a vector (a window closed on both sides),
hundreds of calls on one context: every CTA and warp must take the same window."""
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
@pytest.mark.parametrize("n", [600_011, 3_000_017])
def test_repeated(g, dtype, n):
    r = np.random.default_rng(n)
    x = (r.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) if dtype == np.uint32
         else r.standard_normal(n).astype(dtype))
    desc = np.sort(x)[::-1]
    d = DeviceArray(x)
    ctx = g.Context(0)
    for i in range(120):
        mid = int(r.integers(n // 8, n - n // 8))
        for ks in ([mid], [mid, mid + 5, mid + n // 64]):
            ks = np.array(ks, dtype=np.uint32)
            assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=False), desc[ks - 1],
                        f"call {i}, k's {ks}")
    ctx.close()


@pytest.mark.parametrize("dist", ["normal", "uniform", "crowd"])
def test_crowded_slices(g, dist):
    """Doubles, whose fine slices of the sample are half a binade wide and hold up to a
    quarter of it (all of it: "crowd"): the window stays as narrow as the sample allows."""
    n = 20_000_003
    r = np.random.default_rng(3)
    x = r.standard_normal(n) if dist == "normal" else r.random(n) * 2e6 - 1e6
    if dist == "crowd":
        x = 1000.0 + x * 1e-9
        x[r.choice(n, 2000, replace=False)] = r.random(2000) * 1e300
    desc = np.sort(x)[::-1]
    d = DeviceArray(x)
    ctx = g.Context(0)
    for at in (0.3, 0.45, 0.7, 0.93):
        ks = np.array([int(n * at)], dtype=np.uint32)
        assert_same(g.multiselect_ptr(d.ptr, n, np.float64, ks, ctx=ctx), desc[ks - 1], f"{dist} {at}")
    assert ctx.stats()["topk_misses"] == 0
    for K in (16, 3000, 20000):
        assert_same(g.topk_ptr(d.ptr, n, np.float64, K, ctx=ctx), desc[:K], f"{dist} top-{K}")
    if dist != "crowd":  # (whose top-k's span the gap below the values far out)
        assert ctx.stats()["topk_misses"] == 0
    ctx.close()
