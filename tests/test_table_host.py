"""The splitter table (csrc/ggks_front.cuh, csrc/ggks_device.cuh) built on the host CPU:
buckets ascend with the keys, each begins at its smallest key, and the keys below
the smallest sampled one have a bucket of their own wherever that key lies."""
import ctypes

import numpy as np
import pytest

from test_window_host import emu, keys  # noqa: F401  (the fixture)


def check(emu, x, fn, extra, nb_max=8192):
    k = keys(x)
    top = ~k.dtype.type(0)
    lo, hi = k.min(), k.max()
    probe = np.concatenate([k, extra.astype(k.dtype), np.array([0, 1, top, top - 1], k.dtype)])
    near = np.array([v + d for v in (int(lo), int(hi)) for d in range(-3, 4)
                     if 0 <= v + d <= int(top)], dtype=k.dtype)
    probe = np.unique(np.concatenate([probe, near]))
    bucket = np.zeros(probe.size, np.uint32)
    first = np.zeros(probe.size, k.dtype)
    nb = ctypes.c_uint32()
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert fn(ptr(x), ctypes.c_uint64(x.size), nb_max, ptr(probe), probe.size, ptr(bucket), ptr(first),
              ctypes.byref(nb)) == 0
    assert np.all(np.diff(bucket.astype(np.int64)) >= 0) and bucket[-1] < nb.value <= nb_max
    assert np.all(first <= probe)
    for b in np.unique(bucket):  # a bucket's smallest key lies past the buckets before it
        at = np.flatnonzero(bucket == b)
        assert np.all(first[at] == first[at[0]])
        if at[0]:
            assert first[at[0]] > probe[at[0] - 1]
    return dict(zip(probe.tolist(), bucket.tolist())), int(lo), int(hi)


@pytest.mark.parametrize("lo", [0, 1, 1000, 1 << 20, 1 << 26, 1 << 31])
@pytest.mark.parametrize("span", [1, 300, 65535, 1 << 22, (1 << 31) - 1])
def test_u32(emu, lo, span):  # noqa: F811
    r = np.random.default_rng(span)
    x = (lo + r.integers(0, span + 1, 5000, dtype=np.uint64)).clip(0, (1 << 32) - 1).astype(np.uint32)
    x[:1500] = lo
    x[1500:1502] = min(lo + span, (1 << 32) - 1)
    b, kmin, kmax = check(emu, x, emu.emu_table_u32, r.integers(0, 1 << 32, 3000, dtype=np.uint64))
    assert kmin == lo
    if kmin:
        assert b[kmin - 1] != b[kmin] and b[0] == b[kmin - 1] == 0


def test_u32_whole_range(emu):  # noqa: F811
    """No low entry fits below a table that reaches the largest key."""
    r = np.random.default_rng(1)
    for lo, hi in ((0, 1 << 32), (5, 1 << 32), (1 << 22, 1 << 32), (7, (1 << 32) - 100)):
        x = r.integers(lo, hi, 6000, dtype=np.uint64).astype(np.uint32)
        x[:3] = [lo, hi - 1, hi - 2]
        check(emu, x, emu.emu_table_u32, r.integers(0, 1 << 32, 3000, dtype=np.uint64))


@pytest.mark.parametrize("dist", ["normal", "positive", "few", "special"])
def test_f64(emu, dist):  # noqa: F811
    r = np.random.default_rng(3)
    x = r.standard_normal(6000)
    if dist == "positive":
        x = np.abs(x) * 1e300
    elif dist == "few":
        x = r.integers(-3, 4, 6000) * 1.0
    elif dist == "special":
        x[:40] = np.resize(np.array([np.inf, -np.inf, 0.0, -0.0, np.nan, -np.nan, 5e-324]), 40)
    check(emu, x, emu.emu_table_f64, r.integers(0, 1 << 64, 2000, dtype=np.uint64), 16384)
