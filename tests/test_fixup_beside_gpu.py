"""The fix-up beside the bulk pass (many particles, batches) against the fix-up behind it.

A model's slots are computed by the same code and its momentum exchange is summed in the same order on both ways, so
the states are equal.  A batch's schedules share one CTA shape, so they are
equal too."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # one chunk per particle and several, walked in turn or side by side; both kinds of bulk pass
    "bf16": dict(n=(96, 96, 96), count=64, r=6.0, storage="bf16"),
    "f32_turns": dict(n=(192, 160, 160), count=48, r=7.0),
    "f16_nearest": dict(n=(96, 80, 96), count=48, r=7.0, storage="f16", rounding="nearest"),
    "odd_rows_f64": dict(n=(101, 96, 90), count=48, r=6.5, storage="f64", collision="bgk"),
    "d3q27": dict(n=(96, 96, 96), count=48, r=6.0, lattice="D3Q27"),
    "d2q9": dict(n=(900, 800), count=240, r=24.0, storage="f16"),
    # wall links and nodes in the same list; particles whose near boxes meet the walls and each other
    "walls": dict(n=(96, 80, 96), count=60, r=9.2, walls=True),
    "touching": dict(n=(80, 80, 80), count=64, r=9.4),
}


def _model(case):
    import lbmengine as lbm
    n, c = case["n"], case["count"]
    d = len(n)
    rng = np.random.default_rng(sum(n) + c)
    kw = dict(dims=d, latticeParameter=1.0, relaxationTimeRatio=0.8, collisionModel=case.get("collision", "trt"),
              storage=case.get("storage", "f32"), forceDensity=[1e-6] + [0.0] * (d - 1),
              fluidVelocity=1e-3 * rng.standard_normal((*n, d)))
    if "lattice" in case:
        kw["velocities"] = case["lattice"]
    if "rounding" in case:
        kw["rounding"] = case["rounding"]
    for k, a in zip(n, ("xlims", "ylims", "zlims")):
        kw[a] = (-float(k // 2), float(k - 1 - k // 2))
    if case.get("walls"):
        kw["walledDimensions"] = [2]
    m = lbm.modelInit(**kw)
    g = int(np.ceil(c ** (1 / d) - 1e-9))
    for at in list(np.ndindex(*([g] * d)))[:c]:
        e = rng.standard_normal(d)
        pos = [-n[k] / 2 + (at[k] + 0.5) * n[k] / g + rng.uniform(-0.4, 0.4) for k in range(d)]
        lbm.addSquirmer(m, radius=case["r"], position=pos, massDensity=3.0, swimmingSpeed=2e-3, beta=1.5,
                        swimmingDirection=list(e / np.linalg.norm(e)), coupleForces=True, coupleTorques=True)
    return m


@pytest.mark.parametrize("name", CASES)
def test_same_state_beside_and_behind(name):
    from lbmengine import _capi as capi
    lib = capi.load()
    out = []
    for profiling in (0, 2):  # per-kernel events keep the fix-up behind the bulk pass
        m = _model(CASES[name])
        assert lib.lbm_set_profiling(m.handle, profiling) == 0
        for ticks in (3, 21):
            m.step(ticks)
        launches = capi.LbmProfile()
        lib.lbm_get_profile(m.handle, C.byref(launches))
        p = m.particle_states()
        out.append((launches.launches, m.distributions.copy(),
                    np.concatenate([np.ravel(np.asarray(v, dtype=float)) for q in p
                                    for v in (q.position, q.velocity, q.angular_velocity)])))
        m.close()
    assert [o[0] for o in out] == [21 * 4, 21 * 3]  # the first took the list
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("storage,lattice", [("f32", "D2Q9"), ("f16", "D2Q9"), ("bf16", "D3Q19")])
def test_batch_schedules_agree(storage, lattice, walls):
    import lbmengine as lbm
    d = 2 if lattice == "D2Q9" else 3
    reps = []
    for i, side in enumerate((32, 40, 64, 36)):
        kw = dict(dims=d, velocities=lattice, latticeParameter=1.0, relaxationTimeRatio=0.7 + 0.05 * i,
                  collisionModel="trt", storage=storage, forceDensity=[1e-5] + [0.0] * (d - 1))
        for a in ("xlims", "ylims", "zlims")[:d]:
            kw[a] = (-side / 2, side / 2 - 1)
        if walls and i != 1:
            kw["walledDimensions"] = [2]
        sq = [("squirmer", dict(radius=4.0 + i, position=[s * side / 4.1] + [0.3] * (d - 1), massDensity=3.0,
                                swimmingSpeed=2e-3, beta=2.0, swimmingDirection=[0.6, 0.8] + [0.0] * (d - 2),
                                coupleForces=True, coupleTorques=True)) for s in (-1, 1)[:i % 3]]
        reps.append((kw, sq))
    out = []
    for tuning in (dict(schedule="persistent"), dict(schedule="stream"), dict(schedule="stream", tile_cta=1)):
        b = lbm.LBMbatch(reps)
        b.set_tuning(ctas_per_sm=2, **tuning)
        for ticks in (1, 2, 37):
            b.step(ticks)
        out.append([m.distributions.copy() for m in b.replicas])
        del b
    for other in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(out[0], other))
