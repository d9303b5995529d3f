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


def _swimmer(**kw):
    import lbmengine as lbm
    m = lbm.modelInit(dims=3, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel="trt",
                      xlims=(-10.0, 9.0), ylims=(-10.0, 9.0), zlims=(-10.0, 9.0), **kw)
    lbm.addSquirmer(m, radius=4.0, position=[0.3, 0.1, -0.2], massDensity=2.0, swimmingSpeed=1e-3, beta=2.0,
                    coupleForces=True, coupleTorques=True)
    return m


@pytest.mark.parametrize("extra", [1000, 3_000_000])  # no room for the stored states; for some of the buffers
def test_refused_gradient_gives_its_bytes_back(lib, extra):
    from lbmengine.adjoint import swimming_speed_gradient
    m = _swimmer()
    before = m.info().device_bytes
    with limit(lib, before + extra), pytest.raises(capi.LbmError) as e:
        swimming_speed_gradient(m, 6, (4, 6), snapshots=3)
    assert e.value.code == capi.LBM_ERR_OOM
    assert m.info().device_bytes == before
    out = swimming_speed_gradient(m, 6, (4, 6), snapshots=3)
    assert m.info().device_bytes == before
    assert out.value == swimming_speed_gradient(_swimmer(), 6, (4, 6), snapshots=3).value


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("extra", [16, 24_600])  # no room for any buffer of the many-ticks launch; for the masks alone
def test_small_model_at_the_limit_steps_in_stream_order(lib, walls, extra):
    import lbmengine as lbm

    def model(schedule):
        m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, schedule=schedule,
                          xlims=(-32.0, 31.0), ylims=(-24.0, 23.0), walledDimensions=[2] if walls else [])
        lbm.addSquirmer(m, radius=6.0, position=[0.3, 0.2], massDensity=3.0, swimmingSpeed=1e-3, beta=2.0,
                        swimmingDirection=[0.8, 0.6], coupleForces=True, coupleTorques=True)
        return m

    small, ref = model("auto"), model("stream")
    before = small.info().device_bytes
    with limit(lib, before + extra):
        for n in (3, 40):
            small.step(n)
            ref.step(n)
            assert launches(lib, small) == 3 * n
    assert small.info().device_bytes == before
    np.testing.assert_array_equal(small.distributions, ref.distributions)


def test_gradient_of_many_ticks_needs_no_more_device_memory(lib):
    """The device memory that six ticks' gradient fits into does for a thousand: the particle's history goes to host
    memory where the rest fills the limit, with the same result."""
    from lbmengine.adjoint import swimming_speed_gradient

    def gradient(ticks):
        m = _swimmer(storage="f32")
        out = swimming_speed_gradient(m, ticks, (ticks - 2, ticks), snapshots=3)
        m.close()
        return out

    base = _swimmer().info().device_bytes
    low, high = base, base + (1 << 26)  # refused; enough
    while high - low > 64:
        mid = (low + high) // 2
        with limit(lib, mid):
            try:
                gradient(6)
                high = mid
            except capi.LbmError as e:
                assert e.code == capi.LBM_ERR_OOM
                low = mid
    want = gradient(1000)
    with limit(lib, high):
        got = gradient(1000)
    assert got.value == want.value and got.grad == want.grad
