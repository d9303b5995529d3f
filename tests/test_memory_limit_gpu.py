"""Device buffers that only make a call faster are counted and limited like the model's own (lbm_set_memory_limit,
lbm_info.device_bytes); a model that has no room for them steps without them."""
from __future__ import annotations

import contextlib
import ctypes as C

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def limit(lib, nbytes):
    assert lib.lbm_set_memory_limit(nbytes) == 0
    try:
        yield
    finally:
        lib.lbm_set_memory_limit(0)


def launches(lib, m):
    p = capi.LbmProfile()
    assert lib.lbm_get_profile(m.handle, C.byref(p)) == 0
    return p.launches


def _suspension():
    import lbmengine as lbm
    rng = np.random.default_rng(7)
    m = lbm.modelInit(dims=3, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel="trt", storage="bf16",
                      xlims=(-48.0, 47.0), ylims=(-48.0, 47.0), zlims=(-48.0, 47.0), rounding="nearest")
    for at in np.ndindex(4, 4, 4):
        e = rng.standard_normal(3)
        lbm.addSquirmer(m, radius=6.0, position=[-48 + (k + 0.5) * 24 + 0.3 for k in at], massDensity=3.0,
                        swimmingSpeed=2e-3, beta=1.5, swimmingDirection=list(e / np.linalg.norm(e)),
                        coupleForces=True, coupleTorques=True)
    return m


def test_slot_lists_keep_to_the_limit(lib):
    free, held = _suspension(), _suspension()
    before = held.info().device_bytes
    assert free.info().device_bytes == before
    free.step(5)
    assert launches(lib, free) == 5 * 4  # bulk, list, store, particles
    assert free.info().device_bytes > before
    with limit(lib, before + 4096):
        for _ in range(2):
            held.step(5)
            assert launches(lib, held) == 5 * 3  # the fix-up behind the bulk pass
            assert held.info().device_bytes == before
    free.step(5)
    np.testing.assert_array_equal(held.distributions, free.distributions)
