"""A batch's sample by problem size: eight keys a bucket, at least 1024, whole
vectors below that, 8192 where a candidate window rests on it.  Sizes at those
steps, values that fill one bucket, outliers that the sample misses, vectors off a
16-byte boundary.  Every answer equals sorting."""
import numpy as np
import pytest

from gpu_util import DeviceArray, assert_same

pytestmark = pytest.mark.gpu

SIZES = [1, 1023, 1024, 1025, 1031, 2049, 4097, 8191, 8192, 8193, 32767, 32769, 65537, 262143,
         262145, 600_001]


@pytest.fixture(scope="module")
def g():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ggks
    ggks.lib()
    return ggks


@pytest.mark.parametrize("dtype", [np.float32, np.uint32, np.float64])
@pytest.mark.parametrize("values", ["spread", "few", "outliers", "sorted"])
def test_sizes(g, dtype, values):
    r = np.random.default_rng(11)
    m = max(SIZES)
    if values == "few":
        x = r.integers(0, 7, m).astype(dtype)
    elif dtype == np.uint32:
        x = r.integers(0, 1 << 32, m, dtype=np.uint32)
    else:
        x = r.standard_normal(m).astype(dtype)
    if values == "outliers":
        x = (x / 1000 if dtype != np.uint32 else x // 100000).astype(dtype)
        x[r.integers(0, m, 60)] = 4e9 if dtype == np.uint32 else 1e30
    if values == "sorted":
        x = np.sort(x)
    d = DeviceArray(x, pad_front=1)
    ks = [np.unique(r.integers(1, n + 1, 60)).astype(np.uint32) for n in SIZES]
    want = {n: np.sort(x[:n])[::-1] for n in SIZES}
    got = g.multiselect_batch_ptr([d.ptr] * len(SIZES), SIZES, x.dtype, ks)
    for n, k, o in zip(SIZES, ks, got):
        assert_same(o, want[n][k.astype(np.int64) - 1], f"n={n}")
    Ks = [min(n, 50) for n in SIZES]
    got = g.topk_batch_ptr([d.ptr] * len(SIZES), SIZES, x.dtype, Ks)
    for n, k, o in zip(SIZES, Ks, got):
        assert_same(o, want[n][:k], f"top of {n}")
