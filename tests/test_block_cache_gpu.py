"""Freed device blocks are kept up to 4 GiB in the process, the ones freed longest ago giving way: by the device's free
memory before and after models that do not fit the cache together, in a process of their own."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import PKG, REPO

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import numpy as np
import torch
import lbmengine as lbm

GIB = 1 << 30
slack = GIB // 4

def free():
    return torch.cuda.mem_get_info()[0]

def model(side):  # two population buffers of side^3 x 19 x 4 bytes
    lim = (0.0, side - 1.0)
    return lbm.modelInit(dims=3, velocities="D3Q19", latticeParameter=1.0, relaxationTimeRatio=0.8, xlims=lim,
                         ylims=lim, zlims=lim, storage="f32")

torch.zeros(1, device="cuda")
m = model(32)
m.step(2)
want = m.distributions.copy()
m.close()
a, b = 2 * 256**3 * 76, 2 * 288**3 * 76  # 2.4 and 3.4 GiB
assert a < 4 * GIB and b < 4 * GIB < a + b
start = free()
model(256).close()
print("kept", abs(start - free() - a) < slack)
model(288).close()  # takes the place of the first one's
print("oldest gone", b - slack < start - free() < 4 * GIB + slack)
before = free()
again = model(288)
print("handed out again", abs(before - free()) < slack)
again.close()
other = model(256)
print("new blocks", before - free() > a // 2 - slack)
other.close()
print("bounded", start - free() < 4 * GIB + slack)
m = model(32)
m.step(2)
print("same", np.array_equal(m.distributions, want))
"""


def test_oldest_blocks_give_way(lib):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, REPO]))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.splitlines() == [f"{k} True" for k in ("kept", "oldest gone", "handed out again", "new blocks",
                                                           "bounded", "same")], r.stdout
