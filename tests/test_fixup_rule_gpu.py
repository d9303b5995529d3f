"""Where the fix-up runs beside the bulk pass (four launches a tick) and where behind it (three): D3Q27 only with more
particles than the other velocity sets, and not with FP64 storage."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,storage,n,count,radius,beside", [
    ("D3Q19", "f32", 128, 27, 6.0, True), ("D3Q19", "f64", 96, 64, 5.0, True),
    ("D3Q27", "f32", 128, 27, 6.0, False), ("D3Q27", "f32", 96, 64, 5.0, True), ("D3Q27", "f16", 128, 27, 6.0, False),
    ("D3Q27", "f16", 128, 64, 6.0, True), ("D3Q27", "f64", 96, 64, 5.0, False), ("D3Q27", "f64", 96, 125, 5.0, False)])
def test_launches_per_tick(lib, lattice, storage, n, count, radius, beside):
    import lbmengine as lbm
    lim = (-n / 2, n / 2 - 1)
    m = lbm.modelInit(dims=3, velocities=lattice, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel="trt",
                      storage=storage, xlims=lim, ylims=lim, zlims=lim)
    g = int(np.ceil(count ** (1 / 3) - 1e-9))
    for at in list(np.ndindex(g, g, g))[:count]:
        lbm.addSquirmer(m, radius=radius, position=[-n / 2 + (k + 0.5) * n / g + 0.2 for k in at], massDensity=3.0,
                        swimmingSpeed=1e-4, beta=2.0, coupleForces=True, coupleTorques=True)
    m.step(3)
    p = capi.LbmProfile()
    assert lib.lbm_get_profile(m.handle, C.byref(p)) == 0
    m.close()
    assert p.launches == 3 * (4 if beside else 3)
