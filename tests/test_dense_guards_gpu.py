"""What a dense table cannot hold is noticed while the call runs, and the call is made
again with an ordinary table: one CTA's count of a key past 16 bits (in either half
of a word; the sample accepts the vector), and more keys outside the sampled range
than their list holds."""
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


def run(g, x, ks):
    d = DeviceArray(x)
    ctx = g.Context(0)
    got = g.multiselect_ptr(d.ptr, x.size, x.dtype, ks, ctx=ctx)
    st = ctx.stats()
    ctx.close()
    assert_same(got, np.sort(x)[::-1][ks.astype(np.int64) - 1])
    return st


@pytest.mark.parametrize("value", [30000, 30001])
def test_count_past_16_bits(g, value):
    import torch
    n = 1 << 24
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = np.random.default_rng(1).integers(0, 65536, n).astype(np.uint32)
    # the first CTA's tiles, of 4 or 8 vectors a thread: 1 / sms of the vector
    at = np.arange(n)
    for tile in (1 << 14, 1 << 15):
        x[at // tile % sms == 0] = value
    ks = np.linspace(1, n, 500).astype(np.uint32)
    assert run(g, x, ks)["retries"] == 1


@pytest.mark.parametrize("side", ["below", "above"])
def test_list_overflow(g, side):
    n = (1 << 22) + 3
    r = np.random.default_rng(2)
    x = (1000000 + r.integers(0, 65000, n)).astype(np.uint32)
    free = np.setdiff1d(np.arange(n), np.unique(sampled_positions(n).astype(np.int64)))
    many = 40_000
    out = r.integers(0, 900_000, many) + (3_000_000 if side == "above" else 0)
    x[r.choice(free, many, replace=False)] = out.astype(np.uint32)
    inside = np.linspace(n // 20, n - n // 20, 400).astype(np.uint32)
    st = run(g, x, inside)  # the list is not needed
    assert st["retries"] == 0 and st["survivors"] == 0
    edge = many // 2 if side == "above" else n - many // 2
    assert run(g, x, np.append(inside, np.uint32(edge)))["retries"] == 1
