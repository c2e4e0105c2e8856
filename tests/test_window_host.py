"""The sampled-window kernels (csrc/ggks_window.cuh) run on the host CPU, one block
at a time, with thread 0 as far ahead of the other threads as the barriers allow
(device_emu/cuda_on_host.h): what they write must not depend on how far that is.
Every element is sampled here, so the window's ends are known exactly."""
import ctypes
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "device_emu"))
import build_emu  # noqa: E402

BINS = 8192
DEFERRED, MISS = 2, 32  # ST_DEFERRED, ST_TOPK_MISS
EMPTY = 0xABCDEF01
U32 = ctypes.POINTER(ctypes.c_uint32)


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    lib = build_emu.build("window_kernels.cpp",
                          ["ggks_device.cuh", "ggks_front.cuh", "ggks_tiny.cuh", "ggks_window.cuh"],
                          tmp_path_factory.mktemp("emu"))
    if lib is None:
        pytest.skip("no host compiler or CUDA headers")
    return lib


def keys(x):
    if x.dtype == np.uint32:
        return x.copy()
    u = np.dtype(f"u{x.itemsize}").type
    b, top = x.view(u), u(1 << (8 * x.itemsize - 1))
    return np.where(b & top, ~b, b | top)


def make(dtype, dist, n):
    r = np.random.default_rng(n)
    if dist == "limits":  # the smallest and the largest key, 40 % of the vector each
        u = np.dtype(f"u{np.dtype(dtype).itemsize}")
        top = u.type(-1 % (1 << 8 * u.itemsize)) >> u.type(dtype != np.uint32)
        b = (r.random(n) * 1e9).astype(dtype).view(u)
        p = r.random(n)
        return np.where(p < 0.4, u.type(0 if dtype == np.uint32 else -1 % (1 << 8 * u.itemsize)),
                        np.where(p < 0.8, top, b)).astype(u).view(dtype)
    if dist == "few":
        x = r.integers(0, 5, n) * 100.0
    elif dist == "spread":
        x = r.random(n) * 1e9
    elif dist == "crowd":  # most samples in one fine slice, a few far out
        x = 1000.0 + r.random(n)
        x[r.choice(n, 20, replace=False)] = r.random(20) * 1e9
    elif dist == "same":  # a fine slice of one key
        x = np.where(r.random(n) < 0.97, 1000.0, r.random(n) * 1e9)
    else:
        x = r.standard_cauchy(n) * 1e4
    return (np.abs(x) if dtype == np.uint32 else x).clip(-4e9, 4e9).astype(dtype)


def run_filter(emu, x, r0, r1, lo_open, hi_open, grid=3):
    k = keys(x)
    arr = np.zeros(x.size, k.dtype)
    bins = np.zeros(BINS, np.uint32)
    out = np.zeros(8, np.uint64)
    fn = {np.dtype(np.float32): emu.emu_filter_f32, np.dtype(np.float64): emu.emu_filter_f64,
          np.dtype(np.uint32): emu.emu_filter_u32}[x.dtype]
    rc = fn(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(x.size), r0, r1, int(lo_open),
            int(hi_open), grid, arr.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(x.size),
            bins.ctypes.data_as(U32), out.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0
    return k, arr, bins, [int(v) for v in out]


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
@pytest.mark.parametrize("dist", ["spread", "heavy", "few", "crowd", "same", "limits"])
@pytest.mark.parametrize("ends", ["closed", "low", "high"])
def test_filter(emu, dtype, dist, ends):
    n = 5003 if dist not in ("crowd", "same") else 9001  # (past 4096 in a slice)
    x = make(dtype, dist, n)
    r0, r1 = {"closed": (2300, 2700), "low": (0, 300), "high": (n - 400, n - 1)}[ends]
    lo_open, hi_open = ends == "low", ends == "high"
    k, arr, bins, (length, below, lo, shift, inner, counted, key_lo, key_hi) = run_filter(
        emu, x, r0, r1, lo_open, hi_open)
    s = np.sort(k)
    has_lo, has_hi = counted & 1, counted >> 1
    share = {e: np.count_nonzero(k == s[r]) / n for e, r in (("lo", r0), ("hi", r1))}
    popular = (not lo_open and share["lo"] > 1 / 128) or (not hi_open and share["hi"] > 1 / 128)
    same = ends == "closed" and s[r0] == s[r1]
    assert bool(counted) == (popular or same)
    keep = np.ones(n, bool)
    if not lo_open:
        keep &= k > s[r0] if has_lo else k >= s[r0]
    if not hi_open:
        keep &= k < s[r1] if has_hi else k <= s[r1]
    want = np.sort(k[keep])
    assert length == want.size
    if ends == "closed":
        assert below == np.count_nonzero(k < s[r0])
    assert np.array_equal(np.sort(arr[:length]), want)
    at = [has_lo + (0 if v < lo else min((v - lo) >> shift, inner - 1)) for v in want.tolist()]
    expect = np.bincount(np.array(at, int), minlength=BINS)
    if has_lo:
        assert key_lo == s[r0]
        expect[0] += np.count_nonzero(k == s[r0])
    if has_hi:
        assert key_hi == s[r1]
        expect[has_lo + inner] += np.count_nonzero(k == s[r1])
    assert np.array_equal(bins, expect)


def place(emu, arr, n, below, lo, shift, nbins, bins, kk, ranks, grid, sort=False):
    guard = 64
    placed = np.full(arr.size + guard, EMPTY, np.uint32)
    out = np.full(max(kk, ranks.size), EMPTY, np.uint32)
    status = ctypes.c_uint32()
    rc = emu.emu_place_u32(
        arr.ctypes.data_as(U32), arr.size, ctypes.c_uint64(n), below, lo, shift, nbins,
        bins.ctypes.data_as(U32), kk, ranks.ctypes.data_as(U32), ranks.size, grid,
        placed.ctypes.data_as(U32), ctypes.c_uint64(arr.size),
        out.ctypes.data_as(U32) if sort else None, ctypes.byref(status))
    assert rc == 0, "threads wait for others that never come"
    assert np.all(placed[arr.size:] == EMPTY)
    return placed[:arr.size], out, status.value


@pytest.mark.parametrize("big", ["none", "copies", "distinct"])
def test_topk_bins(emu, big):
    """Bins that a warp sorts, large bins of one key and large bins of many keys, which
    the first CTA leaves to a recursive level while others may still read the status."""
    r = np.random.default_rng(1)
    n, lo, shift, nbins, kk = 100_000, 5000, 6, 300, 3000
    arr = (lo + r.integers(0, nbins << shift, 4000)).astype(np.uint32)
    if big != "none":
        at = nbins - 40 - np.arange(16) * 2
        extra = lo + (np.repeat(at, 400) << shift)
        extra += r.integers(0, 1 << shift, extra.size) if big == "distinct" else 3
        arr = np.concatenate([arr[~np.isin((arr - lo) >> shift, at)], extra]).astype(np.uint32)
    bins = np.bincount((arr - lo) >> shift, minlength=BINS).astype(np.uint32)
    _, out, status = place(emu, arr, n, 0, lo, shift, nbins, bins, kk, np.zeros(0, np.uint32), 3,
                           sort=True)
    want = np.sort(arr)[::-1][:kk]
    assert status == (DEFERRED if big == "distinct" else 0)
    later = np.isin((want - lo) >> shift, at) if big == "distinct" else np.zeros(kk, bool)
    assert np.array_equal(out[~later], want[~later]) and np.all(out[later] == EMPTY)


@pytest.mark.parametrize("big", ["none", "copies", "distinct"])
def test_request_bins(emu, big):
    r = np.random.default_rng(2)
    n, lo, shift, nbins, below = 1_000_000, 5000, 20, 50, 400_000
    arr = (lo + r.integers(0, nbins << shift, 6000)).astype(np.uint32)
    b = 17
    if big != "none":
        extra = lo + (b << shift) + (r.integers(0, 1 << shift, 66_000) if big == "distinct" else 7)
        arr = np.concatenate([arr[(arr - lo) >> shift != b], np.broadcast_to(extra, 66_000)])
        arr = r.permutation(arr.astype(np.uint32))
    s = np.sort(arr)
    bins = np.bincount((arr - lo) >> shift, minlength=BINS).astype(np.uint32)
    local = np.array([0, 3000, 3001, arr.size // 2, arr.size - 1, 3000])
    _, out, status = place(emu, arr, n, below, lo, shift, nbins, bins, 0,
                           (local + below).astype(np.uint32), 2, sort=True)
    want = s[local]
    assert status == (DEFERRED if big == "distinct" else 0)
    later = (want - lo) >> shift == b if big == "distinct" else np.zeros(local.size, bool)
    assert np.array_equal(out[~later], want[~later]) and np.all(out[later] == EMPTY)


@pytest.mark.parametrize("kk", [0, 700])
@pytest.mark.parametrize("grid", [1, 2])
def test_place(emu, kk, grid):
    """Candidates go to the places of their bins; a bin that meets more keys than it
    counted stores none outside its places, and the call is a miss."""
    r = np.random.default_rng(grid)
    n, length, lo, shift, nbins = 100_000, 4500, 1000, 4, 500
    arr = (lo + r.integers(0, nbins << shift, length)).astype(np.uint32)
    at = (arr - lo) >> shift
    true = np.bincount(at, minlength=BINS).astype(np.uint32)
    first = int(np.searchsorted(np.cumsum(true), length - kk, side="right")) if kk else 0
    below = n - length if kk else 40_000
    short = true.copy()  # a needed bin counts two keys too few, a later one two too many
    short[first] -= 2
    short[first + 9] += 2
    ranks = np.zeros(0, np.uint32) if kk else np.array([0, 1000, length - 1], np.uint32) + 40_000
    for bins in (true, short):
        placed, _, status = place(emu, arr, n, below, lo, shift, nbins, bins, kk, ranks, grid)
        assert (status == 0) if bins is true else (status & MISS)
        pre = np.concatenate([[0], np.cumsum(bins)]).astype(int)
        need = range(first, nbins) if kk else np.searchsorted(pre, ranks.astype(int) - below, "right") - 1
        for b in range(nbins):
            part = placed[pre[b]:pre[b + 1]]
            if b not in need:
                assert np.all(part == EMPTY)
            elif bins is true:
                assert np.array_equal(np.sort(part), np.sort(arr[at == b]))
            else:
                assert np.all((part[part != EMPTY] - lo) >> shift == b)


@pytest.mark.parametrize("threads", [64, 1024])
@pytest.mark.parametrize("c", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 500, 1000, 1024, 1025, 3000])
def test_sort_any_length(emu, threads, c):
    r = np.random.default_rng(c)
    guard = 40
    for hi in (3, 1 << 60):
        a = r.integers(0, hi, c + guard).astype(np.uint64)
        a[r.integers(0, c)] = ~np.uint64(0)
        want = np.concatenate([np.sort(a[:c]), a[c:]])
        assert emu.emu_sort_u64(a.ctypes.data_as(ctypes.c_void_p), c, threads) == 0
        assert np.array_equal(a, want)


@pytest.mark.parametrize("kind", ["spread", "crowd", "narrow", "full"])
@pytest.mark.parametrize("size", [257, 1000, 4097, 20_000, 32_768])
def test_big_bin(emu, kind, size):
    """One large bin of a top-k: parts that a thread sorts, a crowded part, parts one key wide."""
    r = np.random.default_rng(size)
    off, above = 37, 100
    keys = {"spread": lambda: r.integers(1 << 20, 1 << 30, size),
            "crowd": lambda: np.append(r.integers(0, 5000, size - 1), 0xFFFFFFFF),
            "narrow": lambda: 7 + r.integers(0, 4000, size),
            "full": lambda: r.permutation(size) * 131}[kind]().astype(np.uint32)
    placed = np.concatenate([np.zeros(off, np.uint32), keys])
    for kk in (above + size, above + size // 3, above + 1):
        out = np.full(above + size + 8, EMPTY, np.uint32)
        rc = emu.emu_big_u32(placed.ctypes.data_as(U32), ctypes.c_uint64(off), size, above, kk,
                             out.ctypes.data_as(U32))
        assert rc == 0
        assert np.array_equal(out[above:kk], np.sort(keys)[::-1][:kk - above])
        assert np.all(out[:above] == EMPTY) and np.all(out[kk:] == EMPTY)
