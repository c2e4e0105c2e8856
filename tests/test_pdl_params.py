"""Kernels launched with programmatic serialization are resident while their
predecessors write what they read: no parameter of one may promise read-only data
(const T *__restrict__), which would let the compiler load it ahead of the wait."""
import glob
import os
import re

import pytest

from conftest import PKG

HEADERS = sorted(glob.glob(os.path.join(PKG, "csrc", "*.cuh")))


def closing(text, at, pair):
    depth = 1
    while depth:
        depth += (text[at] == pair[0]) - (text[at] == pair[1])
        at += 1
    return at


def kernels(text):
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        end = closing(text, m.end(), "()")
        body = text.index("{", end) + 1
        yield m.group(1), text[m.end():end], text[body:closing(text, body, "{}")]


@pytest.mark.parametrize("path", HEADERS, ids=[os.path.basename(p) for p in HEADERS])
def test_no_read_only_promise(path):
    with open(path) as f:
        text = f.read()
    bad = [name for name, params, body in kernels(text)
           if re.search(r"\bpdl_(start|wait)\(", body)
           and re.search(r"const [^,]*?\*\s*__restrict__", params)]
    assert not bad


def test_kernels_are_found():
    names = set()
    for path in HEADERS:
        with open(path) as f:
            names |= {n for n, _, body in kernels(f.read()) if re.search(r"\bpdl_(start|wait)\(", body)}
    assert {"k_sample", "k_hist", "k_compact", "k_finish", "k_wplace", "k_pick"} <= names
