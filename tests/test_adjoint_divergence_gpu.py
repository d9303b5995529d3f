"""A gradient run that diverges: LBM_ERR_NUMERIC, naming the tick at which plain steps fail, also where the divergence
lies in the middle of a segment of the checkpoint schedule."""
from __future__ import annotations

import re

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu


def _model(storage="f32"):
    """A shear layer of supersonic speeds next to tau = 1/2, which a few ticks blow up."""
    import lbmengine as lbm
    n = 24
    y = np.arange(n)
    u = np.zeros((n, n, n, 3))
    u[..., 0] = 0.55 * np.sin(2 * np.pi * y / n)[None, :, None]
    u[..., 1] = 0.05 * np.random.default_rng(3).standard_normal((n, n, n))
    m = lbm.modelInit(dims=3, latticeParameter=1.0, relaxationTimeRatio=0.501, collisionModel="trt", storage=storage,
                      xlims=(-12.0, 11.0), ylims=(-12.0, 11.0), zlims=(-12.0, 11.0), fluidVelocity=u)
    lbm.addSquirmer(m, radius=4.0, position=[0.3, 0.1, -0.2], massDensity=2.0, swimmingSpeed=1e-3, beta=2.0,
                    coupleForces=False, coupleTorques=False)
    return m


@pytest.mark.parametrize("ticks,snapshots", [(60, 4), (60, 61), (300, 5)])
def test_divergence_names_its_tick(lib, ticks, snapshots):
    from lbmengine.adjoint import swimming_speed_gradient
    m = _model()
    tick = None
    for _ in range(50):
        try:
            m.step(1)
        except capi.LbmError as e:
            assert e.code == capi.LBM_ERR_NUMERIC
            tick = m.tick
            break
    assert tick is not None and tick > 2
    m = _model()
    with pytest.raises(capi.LbmError) as e:
        swimming_speed_gradient(m, ticks, (ticks // 2, ticks), snapshots=snapshots)
    assert e.value.code == capi.LBM_ERR_NUMERIC
    named = int(re.search(r"near tick (\d+)", str(e.value)).group(1))
    assert abs(named - tick) <= 1, (named, tick)
