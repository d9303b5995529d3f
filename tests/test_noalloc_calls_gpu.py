"""lbm_step_noalloc calls no allocating routine of the CUDA runtime: counted by a preloaded library that stands
before the runtime's functions, in a process whose first steps are the allocation-free ones."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import PKG, REPO

pytestmark = pytest.mark.gpu

# each forwards to the runtime and adds one to the count
COUNTED = {
    "cudaMalloc": ("void**", "size_t"), "cudaHostAlloc": ("void**", "size_t", "unsigned"),
    "cudaMallocHost": ("void**", "size_t"), "cudaMallocAsync": ("void**", "size_t", "void*"),
    "cudaFree": ("void*",), "cudaFreeHost": ("void*",), "cudaHostRegister": ("void*", "size_t", "unsigned"),
    "cudaGraphInstantiate": ("void*", "void*", "unsigned long long"), "cudaStreamCreate": ("void*",),
    "cudaEventCreate": ("void*",),
}

SCRIPT = r"""
import ctypes as C
import lbmengine as lbm
from lbmengine import _capi as capi
calls = C.CDLL(None).counted_calls
calls.restype = C.c_int
lib = capi.load()
def model(particle):
    m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, xlims=(0.0, 47.0), ylims=(0.0, 39.0))
    if particle:
        lbm.addSquirmer(m, radius=5.0, position=[20.3, 18.2], swimmingSpeed=1e-3, beta=2.0)
    return m
for particle in (False, True, False):
    m = model(particle)
    before = calls()
    for n in (1, 3):
        assert lib.lbm_step_noalloc(m.handle, n) == 0, lib.lbm_last_error(m.handle)
    print("calls", calls() - before)
assert calls() > 0  # the models themselves
"""


def test_no_allocating_call(lib, tmp_path):
    src = ["#define _GNU_SOURCE", "#include <dlfcn.h>", "static int n;", "int counted_calls(void) { return n; }"]
    for name, types in COUNTED.items():
        args = ", ".join(f"{t} a{i}" for i, t in enumerate(types))
        src.append(f"int {name}({args}) {{ static int (*f)({', '.join(types)}); "
                   f"if (!f) f = (int (*)({', '.join(types)}))dlsym(dlopen(\"libcudart.so.12\", RTLD_LAZY | RTLD_NOLOAD), "
                   f"\"{name}\"); ++n; "
                   f"return f({', '.join(f'a{i}' for i in range(len(types)))}); }}")
    (tmp_path / "count.c").write_text("\n".join(src).replace("size_t", "unsigned long") + "\n")
    so = str(tmp_path / "count.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(tmp_path / "count.c"), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=os.pathsep.join([PKG, REPO]))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["calls", "0"] * 3
