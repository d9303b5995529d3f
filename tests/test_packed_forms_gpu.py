"""The vector bulk pass takes the packed collision or the scalar one by CTA size and by grid size; both round every
operation alike, so the populations are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,rounding", [("f16", "nearest"), ("f16", "stochastic"), ("bf16", "nearest"),
                                              ("bf16", "stochastic"), ("f32", "nearest")])
@pytest.mark.parametrize("collision", ["trt", "bgk"])
def test_d3q27_rows_in_ctas_of_512_and_of_fewer_threads(lib, storage, rounding, collision):
    import lbmengine as lbm
    n = (32, 70, 5)  # 8 threads a row: 64 rows a CTA of 512, the second one with 6
    rng = np.random.default_rng(5)
    kw = dict(dims=3, velocities="D3Q27", latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel=collision,
              storage=storage, rounding=rounding, schedule="stream", forceDensity=[1e-5, -2e-5, 3e-5],
              xlims=(0.0, 31.0), ylims=(0.0, 69.0), zlims=(0.0, 4.0), massDensity=1.0 + 0.01 * rng.standard_normal(n),
              fluidVelocity=0.02 * rng.standard_normal(n + (3,)))
    out = []
    for threads in (512, 128, 32):
        m = lbm.modelInit(**kw)
        assert lib.lbm_set_bulk_kernel(m.handle, capi.LBM_BULK_VECTOR, threads, 0) == 0
        m.step(5)
        out.append(m.distributions.copy())
        m.close()
    for other in out[1:]:
        np.testing.assert_array_equal(out[0], other)


def test_d2q9_bgk_beyond_l2_equals_its_half(lib):
    """1916 x 1918 nodes of 36 bytes lie beyond 126 MB; the same flow with twice the period, in half of them, does not."""
    import lbmengine as lbm
    nx, ny = 1916, 959
    rng = np.random.default_rng(6)
    rho, u = 1.0 + 0.01 * rng.standard_normal((nx, ny)), 0.02 * rng.standard_normal((nx, ny, 2))
    out = []
    for copies in (1, 2):
        m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel="bgk", storage="f32",
                          schedule="stream", xlims=(0.0, nx - 1.0), ylims=(0.0, copies * ny - 1.0),
                          massDensity=np.concatenate([rho] * copies, axis=1),
                          fluidVelocity=np.concatenate([u] * copies, axis=1))
        m.step(6)
        out.append(m.distributions.copy())
        m.close()
    half, whole = out
    assert whole.shape == (nx, 2 * ny, 9)
    np.testing.assert_array_equal(whole, np.concatenate([half, half], axis=1))
