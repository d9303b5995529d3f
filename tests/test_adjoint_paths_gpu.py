"""The adjoint's launch paths against the dual-number oracle: runs long enough to replay graphs for their forward
ticks, and link lists longer than one round of the link kernel (296 CTAs of eight entries).  FP64 storage, the
tolerance of test_adjoint_gpu.py's dual-number comparison."""
from __future__ import annotations

import pytest

from test_adjoint_gpu import CASES, dual_gradient, gpu_gradient

pytestmark = pytest.mark.gpu

PATHS = {
    "graphs": dict(CASES["d2q9_bgk"], ticks=300, window=(100, 300)),
    "long_link_list": dict(
        model=dict(dims=3, velocities="D3Q19", collisionModel="trt", kineticParameter=3 / 16, latticeParameter=1.0,
                   relaxationTimeRatio=0.8, xlims=(-20.0, 19.0), forceDensity=[2e-5, 0.0, 0.0]),
        squirmer=dict(radius=14.5, position=[0.3, -0.2, 0.1], swimmingSpeed=2e-3, beta=2.0,
                      swimmingDirection=[0.6, 0.64, 0.48], coupleForces=True, coupleTorques=True, massDensity=2.0),
        ticks=12, window=(4, 12)),
}


@pytest.mark.parametrize("name", list(PATHS))
def test_adjoint_path_matches_dual_numbers(lib, oracle_mod, name):
    case = PATHS[name]
    J, dJ = dual_gradient(oracle_mod, case)
    out = gpu_gradient(case, "f64", snapshots=6)
    assert abs(out.value - J) <= 1e-10 * abs(J)
    scale = max(abs(v) for v in dJ.values())
    for k, v in dJ.items():
        assert abs(out.grad[k] - v) <= 1e-6 * abs(v) + 1e-9 * scale, f"{k}: adjoint {out.grad[k]:.9e} dual {v:.9e}"
