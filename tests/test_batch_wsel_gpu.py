"""Mid-size slots finished by CTAs or by warps, around the count per CTA of the grid
from which the warps take them (12 for 4-byte keys, 16 for 8-byte ones), with
spread keys and with clusters whose bins do not fit a warp's buffer.  Every answer
equals sorting."""
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


@pytest.mark.parametrize("dtype,per", [(np.float32, 11), (np.float32, 12), (np.float32, 13), (np.uint32, 12),
                                       (np.float64, 15), (np.float64, 16), (np.float64, 17)])
@pytest.mark.parametrize("cluster", [False, True])
def test_around_the_step(g, dtype, per, cluster):
    import torch
    n, count = 1 << 20, 4
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    r = np.random.default_rng(per)
    x = (r.integers(0, 1 << 32, n, dtype=np.uint32) if dtype == np.uint32
         else r.standard_normal(n).astype(dtype))
    if cluster:
        x[r.permutation(n)[:9000]] = x[0]
        x[r.permutation(n)[:700]] = np.nextafter(x[0], x[0] + 1) if dtype != np.uint32 else x[0] + 1
    want = np.sort(x)[::-1]
    ks = [r.permutation(n)[:per * ctas // count].astype(np.uint32) + 1 for _ in range(count)]
    d = DeviceArray(x)
    got = g.multiselect_batch_ptr([d.ptr] * count, [n] * count, x.dtype, ks)
    for k, o in zip(ks, got):
        assert_same(o, want[k.astype(np.int64) - 1], f"{per} a CTA")
