"""Compiles kernels of csrc/ for the host CPU under cuda_on_host.h.

Copies of the headers are made in which inline PTX is replaced by what it does there
(streaming loads and predicated stores are plain ones, waits on an earlier kernel
do nothing) and dynamic shared memory comes from the launch; nothing else of
the kernels changes."""
import ctypes
import os
import re
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
CSRC = os.path.join(ROOT, "ggks-multiselect_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def _without_asm(text):
    out, at = [], 0
    for m in re.finditer(r"asm volatile\(", text):
        if m.start() < at:
            continue
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if quoted:
                i += c == "\\"
                quoted = c != '"'
            elif c == '"':
                quoted = True
            else:
                depth += (c == "(") - (c == ")")
            i += 1
        code = text[m.start():i]
        out.append(text[at:m.start()])
        out.append("v = *p" if "no_allocate" in code else
                   "if (pred) *p = v" if "@q st.global" in code else "(void)0")
        at = i
    return "".join(out) + text[at:]


def host_source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = _without_asm(f.read())
    return text.replace("extern __shared__ uint4 smem_raw[];",
                        "uint4 *smem_raw = emu::dynamic_smem();")


def build(unit, headers, folder):
    """The shared library of a unit beside this file, built in `folder`; None without
    a host compiler or CUDA's headers."""
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        return None
    for h in headers:
        with open(os.path.join(folder, h), "w") as f:
            f.write(host_source(h))
    lib = os.path.join(folder, "libemu.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w", "-I", str(folder),
                        "-I", HERE, "-I", CUDA_INC, os.path.join(HERE, unit), "-o", lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return ctypes.CDLL(lib)
