"""Device memory that a fresh context takes for calls which need no histogram rows: a
top-k by a threshold and one k by a window.  (2^22 floats: candidates 12 MB, the
sample and tables 2 MB, with room to grow; the rows would be another 40 MB.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["threshold", "window"])
def test_no_rows(what):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    n = 1 << 22
    x = torch.rand(n, device="cuda")
    want = torch.sort(x, descending=True).values[[0, 1023, n // 2 - 1]].cpu().numpy()
    ggks.topk(x, 3)  # the kernels are loaded
    ggks.multiselect(x, np.array([n // 2], np.uint32))
    ctx = ggks.Context(0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    if what == "threshold":
        got = ggks.topk_ptr(x.data_ptr(), n, np.float32, 1024, ctx=ctx)
        assert got[0] == want[0] and got[1023] == want[1]
    else:
        got = ggks.multiselect_ptr(x.data_ptr(), n, np.float32, np.array([n // 2], np.uint32), ctx=ctx)
        assert got[0] == want[2]
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20
    ctx.close()
