"""Many ticks per launch (the default schedule of small 2D models) against the stream schedule.

Both run the same arithmetic per node, link slot and particle and sum the momentum exchange in the same order, so
the runs differ at most by FP64 rounding of the particle update that the compiler may contract differently (1e-12
of the state) and by what that changes in the stored populations (a unit in the last place: 1e-7 with FP32, 1e-13
with FP64).  Solid masks and link lists are equal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SQ = dict(radius=6.0, position=[0.3, 0.2], massDensity=3.0, swimmingSpeed=1e-3, beta=2.0, swimmingDirection=[0.8, 0.6],
          coupleForces=True, coupleTorques=True)
LID = dict(walledDimensions=[2])
CASES = {
    # one cluster of 8, one of 16, a grid; one node per thread and several; odd rows
    "cluster8": dict(n=(48, 40)), "cluster16": dict(n=(89, 71)), "grid": dict(n=(130, 111)),
    "several_nodes_per_thread": dict(n=(301, 400), ticks=(1, 2, 20)),
    "bgk_f64": dict(n=(96, 50), storage="f64", collision="bgk"), "f64_grid": dict(n=(150, 99), storage="f64"),
    "cpu_rules": dict(n=(64, 48), rules="cpu"),
    # the box of the particle moves on by a node in both axes within the run
    "box_moves": dict(n=(64, 64), sq=dict(position=[0.4995, 0.4996]), ticks=(7, 40, 41)),
    # clipped at the domain's edge: the full update in every tick, links across the periodic boundary
    "clipped": dict(n=(64, 48), sq=dict(position=[-28.2, 0.1])),
    # more link entries than one chunk, than two, and than eight
    "chunks": dict(n=(128, 96), sq=dict(radius=14.5)), "many_chunks": dict(n=(300, 260), sq=dict(radius=45.0), ticks=(1, 6)),
    "held": dict(n=(64, 64), sq=dict(coupleForces=False, coupleTorques=False)),
    "walls": dict(n=(40, 33), walls=True), "walls_bead": dict(n=(201, 65), walls=True, kind="bead"),
    # a particle that overlaps the moving wall: slots that are wall links too
    "overlaps_lid": dict(n=(64, 33), walls=True, lid=True, sq=dict(position=[0.3, 11.2]), ticks=(1, 3, 12)),
    "walls_only": dict(n=(61, 40), walls=True, lid=True, kind=None), "fluid": dict(n=(64, 64), kind=None),
    # a bulk phase longer than the boundary work, with the geometry changing under it
    "long_bulk": dict(n=(700, 640), sq=dict(position=[0.499, 0.4996], swimmingSpeed=5e-3), ticks=(1, 40, 41)),
    # several particles: bonded and repelling; two that come close end the launch; two apart
    "bonded": dict(n=(120, 90), parts=[[-20.3, 0.2], [14.1, 0.6], [0.2, 27.4]], bonds=True),
    "come_close": dict(n=(96, 64), parts=[[-9.6, 0.0], [9.4, 0.3]], toward=True, ticks=(1, 60, 61)),
    "touching": dict(n=(96, 64), parts=[[-7.2, 0.0], [7.4, 0.3]], ticks=(1, 20)),
    "force": dict(n=(64, 40), force=[1e-5, 2e-6]), "force_field": dict(n=(65, 40), force="field"),
}


def _model(case, schedule):
    import lbmengine as lbm
    nx, ny = case["n"]
    rng = np.random.default_rng(nx * ny)
    kw = dict(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel=case.get("collision", "trt"),
              storage=case.get("storage", "f32"), particleRules=case.get("rules", "gpu"), schedule=schedule,
              xlims=(-float(nx // 2), float(nx - 1 - nx // 2)), ylims=(-float(ny // 2), float(ny - 1 - ny // 2)),
              fluidVelocity=1e-3 * rng.standard_normal((nx, ny, 2)))
    if case.get("walls"):
        kw["walledDimensions"] = [2]
        if case.get("lid"):
            top = float(ny - 1 - ny // 2)
            kw["movingWalls"] = lambda x, y: [1e-3, 0.0] if y >= top else [0.0, 0.0]
    force = case.get("force")
    if force is not None:
        kw["forceDensity"] = 1e-5 * rng.standard_normal((nx, ny, 2)) if force == "field" else force
    m = lbm.modelInit(**kw)
    kind = case.get("kind", "squirmer")
    p = dict(SQ, **case.get("sq", {}))
    if "parts" in case:
        for k, pos in enumerate(case["parts"]):
            e = [1.0 - 2.0 * k, 0.0] if case.get("toward") else [0.8, 0.6]
            lbm.addSquirmer(m, **dict(p, position=pos, swimmingDirection=e, swimmingSpeed=8e-3 if case.get("toward") else 1e-3))
        if case.get("bonds"):
            lbm.addLinearBond(m, 1, 2, equilibriumDisplacement=36.0, stiffness=1e-2)
            lbm.addPolarBond(m, 1, 3, 2, stiffness=1e-2)
            lbm.addWCA(m)
        return m
    if kind == "bead":
        p = {k: v for k, v in p.items() if k not in ("swimmingSpeed", "beta", "swimmingDirection")}
        lbm.addBead(m, velocity=[1e-3, -5e-4], **p)
    elif kind:
        lbm.addSquirmer(m, **p)
    return m


@pytest.mark.parametrize("name", list(CASES))
def test_resident_matches_stream(lib, name):
    case = CASES[name]
    a, b = _model(case, "auto"), _model(case, "stream")
    tol = 1e-13 if case.get("storage") == "f64" else 1e-7
    for k, ticks in enumerate(case.get("ticks", (1, 30, 33))):
        for m in (a, b):
            if k == 1:
                m._lib.lbm_record_trajectories(m.handle, 64)
            m.step(ticks)
        np.testing.assert_allclose(a.distributions, b.distributions, rtol=0, atol=tol)
        for p, q in zip(a.particle_states(), b.particle_states()):
            for f in ("position", "velocity", "angular_velocity", "swimming_direction", "last_force", "last_torque"):
                u, v = np.array(getattr(p, f)), np.array(getattr(q, f))
                scale = max(1.0 if f in ("position", "swimming_direction") else 1e-3, float(np.abs(v).max()))
                assert np.abs(u - v).max() <= 1e-12 * scale + (1e-9 if tol > 1e-10 else 0) * scale, (f, u, v)
        for pid in range(1, len(a.particle_states()) + 1):
            np.testing.assert_array_equal(a.solid_region(pid), b.solid_region(pid))
            for u, v in zip(a.boundary_links(pid), b.boundary_links(pid)):
                np.testing.assert_array_equal(u, v)
    a.close()
    b.close()
