"""The one-launch path's middle segments (more keys than a warp sorts, at most 4096,
at most four requests), selected by one warp: spread keys, whose needed bins fit
the warp's buffer, and clusters that fill one bin, which go to the whole CTA; at
the sizes where the kinds of segments change.  Every answer equals sorting."""
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
@pytest.mark.parametrize("extra", [257, 513, 4000, 4097, 9000])
@pytest.mark.parametrize("step", [0, 1, 40])
def test_cluster_few_requests(g, dtype, extra, step):
    """extra keys, step representable values apart, inside one bucket; one to five
    requests fall on them and one on the rest."""
    n = 300_007
    r = np.random.default_rng(extra + step)
    u = np.uint64 if dtype == np.float64 else np.uint32
    x = (r.integers(0, 1 << 32, n, dtype=np.uint32) if dtype == np.uint32
         else r.random(n).astype(dtype))
    one = np.array([1 << 31 if dtype == np.uint32 else 0.5], dtype).view(u)[0]
    x[r.permutation(n)[:extra]] = (one + np.arange(extra, dtype=u) * u(step)).view(dtype)
    want = np.sort(x)[::-1]
    at = int(np.searchsorted(-want.astype(np.float64), -float(np.array([one], u).view(dtype)[0]), "right"))
    d = DeviceArray(x)
    for m in (1, 4, 5):
        ks = np.unique(np.concatenate([np.linspace(at - extra + 2, at - 1, m), [7, n - 5]])).astype(np.uint32)
        got = g.multiselect_ptr(d.ptr, n, x.dtype, ks)
        assert_same(got, want[ks.astype(np.int64) - 1], f"{extra} x {step}, {m} requests")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dist", ["uniform", "normal", "exponential"])
def test_many_ks_of_the_largest_vector(g, dtype, dist):
    n = 1 << 20
    r = np.random.default_rng(9)
    x = {"uniform": r.random, "normal": r.standard_normal, "exponential": r.standard_exponential}[dist](n)
    x = x.astype(dtype)
    ks = np.unique(r.integers(1, n + 1, 1001)).astype(np.uint32)
    d = DeviceArray(x)
    got = g.multiselect_ptr(d.ptr, n, x.dtype, ks)
    assert_same(got, np.sort(x)[::-1][ks.astype(np.int64) - 1], dist)
