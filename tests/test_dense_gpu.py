"""Integer vectors whose values span between 2^15 and 2^16 keys (16-bit data): every
key is a bucket with a 16-bit count.  The ranges' edges, ranges at either end of
the keys, values outside the sampled range (with and without requests there), one
value too frequent for a 16-bit count, and ragged sizes.  Every answer equals sorting; survivors tell which way was taken."""
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


def run(g, x, ks, pad=0):
    n = x.size
    d = DeviceArray(x, pad_front=pad)
    ctx = g.Context(0)
    got = g.multiselect_ptr(d.ptr, n, x.dtype, ks, ctx=ctx)
    assert_same(got, np.sort(x)[::-1][ks.astype(np.int64) - 1])
    s = ctx.stats()
    ctx.close()
    return s


def spread(n, m=300):
    return np.unique(np.concatenate([[1, 2, n - 1, n], np.linspace(1, n, m)]).astype(np.uint32))


@pytest.mark.parametrize("lo,span", [(0, 65535), (0, 65534), (1, 65535), (77, 40000), (0, 32768),
                                     (1 << 31, 50000), ((1 << 32) - 65536, 65535),
                                     ((1 << 32) - 40000, 39999), (12345, 32767), (5, 65536)])
@pytest.mark.parametrize("n,pad", [((1 << 20) + 1, 0), ((1 << 22) + 12345, 3)])
def test_ranges(g, lo, span, n, pad):
    r = np.random.default_rng(span)
    x = (lo + r.integers(0, span + 1, n, dtype=np.uint64)).astype(np.uint32)
    x[r.integers(0, n, 2000)] = lo
    x[r.integers(0, n, 2000)] = lo + span
    s = run(g, x, spread(n), pad)
    if 32768 <= span <= 65535:
        assert s["survivors"] == 0 and s["retries"] == 0
    run(g, x, np.array([1, 7, n - 3, n], np.uint32), pad)


@pytest.mark.parametrize("side", ["below", "above", "both"])
@pytest.mark.parametrize("many", [2, 40])
def test_keys_outside_the_sampled_range(g, side, many):
    """Listed in the histogram pass; ranks that fall on them come from the lists."""
    n = (1 << 21) + 7
    r = np.random.default_rng(3)
    x = (1000000 + r.integers(0, 65000, n)).astype(np.uint32)
    at = r.permutation(n)[:2 * many]
    at[0], at[many] = 0, n - 1  # in the scalar ends of a slice off a 16-byte boundary
    if side != "above":
        x[at[:many]] = np.resize([3, 70000, 5, 3], many)
    if side != "below":
        x[at[many:]] = np.resize([0xFFFFFFFF, 1 << 31, 0xFFFFFFFF, 3000000], many)
    edge = np.concatenate([np.arange(1, 60), np.arange(n - 58, n + 1)])
    ks = np.unique(np.concatenate([edge, np.linspace(1, n, 300)])).astype(np.uint32)
    run(g, x, np.linspace(n // 20, n - n // 20, 400).astype(np.uint32), 1)
    run(g, x, ks, 1)  # (an ordinary table where the sample meets one of them)


def test_lists_are_used(g):
    """One key far out on each side: the sample (1 key in 32) misses both in most
    vectors, and nothing is compacted there."""
    n = (1 << 21) + 7
    listed = 0
    for seed in range(8):
        r = np.random.default_rng(seed)
        x = (1000000 + r.integers(0, 65000, n)).astype(np.uint32)
        at = r.integers(n // 4, n // 2, 2)
        x[at] = [3, 0xFFFFFFFF]
        s = run(g, x, spread(n))
        listed += s["survivors"] == 0 and s["retries"] == 0
    assert listed > 0


@pytest.mark.parametrize("share", [0.002, 0.3, 0.9])
def test_frequent_value(g, share):
    n = (1 << 23) + 5
    r = np.random.default_rng(4)
    x = r.integers(0, 65536, n).astype(np.uint32)
    x[r.random(n) < share] = 40000
    run(g, x, spread(n, 700))
    run(g, np.sort(x), spread(n, 700))
