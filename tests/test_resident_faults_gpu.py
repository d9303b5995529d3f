"""The bounded wait at the grid-wide barrier of the many-ticks launch (small 2D models beyond one cluster): a wait
target that no count reaches, with a short poll limit, ends the launch with LBM_ERR_TIMEOUT; launches of the same call
behind it do nothing; the handle goes on from a checkpoint as a fresh model does."""
from __future__ import annotations

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu


def _model(parts, walls=False):
    import lbmengine as lbm
    m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, xlims=(-65.0, 64.0), ylims=(-55.0, 55.0),
                      walledDimensions=[2] if walls else [], forceDensity=[1e-6, 0.0])
    for k in range(parts):
        lbm.addSquirmer(m, radius=6.0, position=[0.3 + 40.0 * k, 0.2], massDensity=3.0, swimmingSpeed=1e-3, beta=2.0,
                        swimmingDirection=[0.8, 0.6], coupleForces=True, coupleTorques=True)
    return m


@pytest.mark.parametrize("parts,walls", [(0, True), (1, False), (1, True), (2, False)])
@pytest.mark.parametrize("ticks", [10, 9000])  # one launch; three
def test_barrier_gives_up_with_timeout(lib, tmp_path, parts, walls, ticks):
    m = _model(parts, walls)
    m.step(10)
    path = str(tmp_path / "state.lbm")
    m.save_state(path)
    assert lib.lbm_set_wait_limit(m.handle, 2000, 1) == 0
    with pytest.raises(capi.LbmError) as e:
        m.step(ticks)
    assert e.value.code == capi.LBM_ERR_TIMEOUT
    assert lib.lbm_set_wait_limit(m.handle, 1 << 22, 0) == 0
    m.load_state(path)
    m.step(10)
    ref = _model(parts, walls)
    ref.step(20)
    np.testing.assert_array_equal(m.distributions, ref.distributions)
    for p, q in zip(m.particle_states(), ref.particle_states()):
        assert list(p.position) == list(q.position) and list(p.velocity) == list(q.velocity)
    m.close()
    ref.close()


def test_recovery_without_new_limits(lib, tmp_path):
    """The masks of a launch that gave up are cleared by the error itself: the same short limit, which ordinary
    waits of this grid may exceed or not, is kept, and only the state is loaded again."""
    m = _model(1)
    m.step(5)
    path = str(tmp_path / "state.lbm")
    m.save_state(path)
    assert lib.lbm_set_wait_limit(m.handle, 1, 0) == 0
    for _ in range(20):  # a limit of one poll gives up sooner or later
        try:
            m.step(50)
        except capi.LbmError as e:
            assert e.code == capi.LBM_ERR_TIMEOUT
            m.load_state(path)
    assert lib.lbm_set_wait_limit(m.handle, 1 << 22, 0) == 0
    m.load_state(path)
    m.step(20)
    ref = _model(1)
    ref.step(25)
    np.testing.assert_array_equal(m.distributions, ref.distributions)
