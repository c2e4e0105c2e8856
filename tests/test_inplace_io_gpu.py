"""Where requests and results change between pinned host memory read and
written by the kernels in place (at most 1024 requests, at most 4096 results)
and copies on the stream: both sides of each limit, for multiselects and
pipeline top-k's, into host and device outputs, on one context whose pinned
buffer grows and is reused."""
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
@pytest.mark.parametrize("count", [1, 1023, 1024, 1025, 4095, 4096, 4097, 9000, 3])
def test_in_place_limits(g, dtype, count):
    import torch
    n = 300_007
    r = np.random.default_rng(count)
    x = (r.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) if dtype == np.uint32
         else r.standard_normal(n).astype(dtype))
    want = np.sort(x)[::-1]
    ks = r.integers(1, n + 1, count).astype(np.uint32)
    d = DeviceArray(x)
    ctx = g.Context(0)
    for _ in range(2):
        assert_same(g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=False), want[ks - 1],
                    f"{count} k's")
        assert_same(g.topk_ptr(d.ptr, n, dtype, count, ctx=ctx, pipeline=True), want[:count],
                    f"top-{count}, pipeline")
        assert_same(g.topk_ptr(d.ptr, n, dtype, count, ctx=ctx), want[:count], f"top-{count}")
    out = torch.zeros(count + 1, dtype={4: torch.int32, 8: torch.int64}[np.dtype(dtype).itemsize],
                      device="cuda")
    torch.cuda.synchronize()
    g.multiselect_ptr(d.ptr, n, dtype, ks, ctx=ctx, small=False, out_device_ptr=out.data_ptr())
    got = out.cpu().numpy()
    assert got[count] == 0
    assert_same(got[:count].view(dtype), want[ks - 1], f"{count} k's, device output")
    ctx.close()
