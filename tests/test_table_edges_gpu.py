"""The splitter table's ends: keys below the sampled smallest one and above the
sampled largest (a few outliers that the sample hardly ever meets), spans that
begin within the first slice's width of key 0 or end at the largest key, spans
of a few keys (no shift at all) and of every key, and their 8-byte forms.
Every answer equals sorting by the order-preserving key, in the streaming
pipeline, in one launch and in a batch."""
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


def make(shape, dtype, n):
    """Unsigned keys of dtype's width, then viewed as dtype's values."""
    r = np.random.default_rng(n)
    bits = np.dtype(dtype).itemsize * 8
    u = np.uint64 if bits == 64 else np.uint32
    top = (1 << bits) - 1
    if shape == "all":
        k = r.integers(0, top, n, dtype=u, endpoint=True)
    elif shape == "from_zero":
        k = r.integers(0, top // 3, n, dtype=u)
    elif shape == "to_top":
        k = u(top) - r.integers(0, top // 3, n, dtype=u)
    elif shape == "first_slice":  # the span begins below one slice's width
        k = r.integers(3, top // 700, n, dtype=u)
    elif shape == "two_keys":
        k = u(top // 2) + r.integers(0, 2, n, dtype=u)
    else:  # a narrow middle and 20 keys far out on each side
        k = u(top // 2) + r.integers(0, 1 << 22, n, dtype=u)
        at = r.permutation(n)[:40]
        k[at[:20]] = r.integers(0, 1000, 20, dtype=u)
        k[at[20:]] = u(top) - r.integers(0, 1000, 20, dtype=u)
    if np.dtype(dtype).kind != "f":
        return k.astype(dtype)
    sign = u(1 << (bits - 1))
    return np.where(k & sign, k ^ sign, ~k).view(dtype)  # key -> float


def key_sorted(x):
    if x.dtype.kind != "f":
        return np.sort(x)
    u = np.uint64 if x.itemsize == 8 else np.uint32
    b = x.view(u)
    sign = u(1 << (x.itemsize * 8 - 1))
    return x[np.argsort(np.where(b & sign, ~b, b | sign), kind="stable")]


@pytest.mark.parametrize("dtype", [np.uint32, np.float32, np.float64])
@pytest.mark.parametrize("shape", ["all", "from_zero", "to_top", "first_slice", "two_keys", "outliers"])
@pytest.mark.parametrize("n", [40001, (1 << 21) + 5])
def test_table_ends(g, shape, dtype, n):
    x = make(shape, dtype, n)
    want = key_sorted(x)
    ks = np.unique(np.concatenate([np.arange(1, 31), np.linspace(1, n, 400),
                                   np.arange(n - 30, n + 1)]).astype(np.uint32))
    d = DeviceArray(x)
    for small in (True, False):
        ctx = g.Context(0)
        got = g.multiselect_ptr(d.ptr, n, x.dtype, ks, ctx=ctx, small=small)
        assert_same(got, want[n - ks.astype(np.int64)], f"{shape} {n} small={small}")
        ctx.close()
    got = g.multiselect_batch_ptr([d.ptr, d.ptr], [n, n // 2], x.dtype, [ks, ks[:100]])
    assert_same(got[0], want[n - ks.astype(np.int64)], f"batch {shape} {n}")
    half = key_sorted(x[:n // 2])
    assert_same(got[1], half[n // 2 - ks[:100].astype(np.int64)], f"batch {shape} {n // 2}")
