"""Which schedule a small 2D model's calls take, by the kernel launches that the profile counts: one launch for many
ticks, more where a launch ends early or a call has more ticks than one launch takes, none of them where the stream
schedule was asked for."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from lbmengine import _capi as capi

pytestmark = pytest.mark.gpu

MAX_TICKS = 4096  # ticks per launch


def _model(n, parts, schedule="auto", walls=False, toward=False, storage="f32"):
    import lbmengine as lbm
    nx, ny = n
    m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, schedule=schedule, storage=storage,
                      xlims=(-float(nx // 2), float(nx - 1 - nx // 2)), ylims=(-float(ny // 2), float(ny - 1 - ny // 2)),
                      walledDimensions=[2] if walls else [])
    for k, pos in enumerate(parts):
        lbm.addSquirmer(m, radius=6.0, position=pos, massDensity=3.0, swimmingSpeed=8e-3 if toward else 1e-3, beta=2.0,
                        swimmingDirection=[1.0 - 2.0 * k, 0.0] if toward else [0.8, 0.6], coupleForces=True,
                        coupleTorques=True)
    return m


def _launches(lib, m, ticks):
    m.step(ticks)
    p = capi.LbmProfile()
    assert lib.lbm_get_profile(m.handle, C.byref(p)) == 0
    return p.launches


ONE = [[0.3, 0.2]]
APART = [[-20.3, 0.2], [20.1, 0.6]]
TOUCHING = [[-7.2, 0.0], [7.4, 0.3]]


@pytest.mark.parametrize("n,parts,walls", [((48, 40), ONE, False), ((130, 111), ONE, False), ((201, 65), ONE, True),
                                           ((61, 40), [], True), ((64, 64), [], False), ((120, 90), APART, False)])
def test_one_launch_per_call(lib, n, parts, walls):
    m = _model(n, parts, walls=walls)
    assert [_launches(lib, m, t) for t in (10, 30, MAX_TICKS)] == [1, 1, 1]
    assert _launches(lib, _model(n, parts, "stream", walls), 30) == 30 * (1 + bool(parts or walls) + bool(parts))


@pytest.mark.parametrize("n,parts", [((48, 40), ONE), ((130, 111), ONE), ((120, 90), APART)])
def test_more_ticks_than_one_launch_takes(lib, n, parts):
    """From both buffers: after an even and an odd number of ticks.  FP32 populations agree with the stream schedule to
    a unit in the last place per tick at most, which the flow damps: 1e-6 after some thousand ticks."""
    for first in (10, 11):
        a, b = _model(n, parts), _model(n, parts, "stream")
        for ticks in (first, MAX_TICKS + 5, 2 * MAX_TICKS + 1):
            assert _launches(lib, a, ticks) == (ticks + MAX_TICKS - 1) // MAX_TICKS
            b.step(ticks)
        assert a.tick == b.tick
        np.testing.assert_allclose(a.distributions, b.distributions, rtol=0, atol=1e-6)
        for p, q in zip(a.particle_states(), b.particle_states()):
            np.testing.assert_allclose(list(p.position), list(q.position), rtol=0, atol=1e-6)


def test_a_launch_that_ends_early_is_counted_with_what_follows(lib):
    # boxes of index ranges 30..45 and 51..66; the launch ends where the first one's end + 4 reaches the second one's
    # start, after 0.2 and 0.4 nodes of approach
    m, ref = (_model((96, 64), [[-10.2, 0.0], [10.4, 0.3]], s, toward=True) for s in ("auto", "stream"))
    assert _launches(lib, m, 10) == 1
    n = _launches(lib, m, 600)  # one launch, then three per tick
    assert n > 1 and (n - 1) % 3 == 0 and n < 1 + 3 * 600
    ref.step(10)
    ref.step(600)
    np.testing.assert_allclose(m.distributions, ref.distributions, rtol=0, atol=1e-6)
    touching = _model((96, 64), TOUCHING)
    assert _launches(lib, touching, 20) == 1 + 3 * 20  # at the first barrier


def test_close_particles_do_not_pay_for_an_attempt_per_call(lib):
    """After a launch that ended at its first barrier 64 ticks run in stream order before the next attempt, then 128;
    particles that are moved apart are tried at once.  Calls of 8 ticks: three launches a tick, one of an attempt."""
    m, ref = (_model((96, 64), TOUCHING, s) for s in ("auto", "stream"))
    calls = [_launches(lib, m, 8) for _ in range(8 + 16 + 1)]
    assert [k for k, n in enumerate(calls) if n != 24] == [0, 8, 24]
    assert all(n == 25 for n in (calls[0], calls[8], calls[24]))
    for _ in range(len(calls)):
        ref.step(8)
    np.testing.assert_array_equal(m.distributions, ref.distributions)
    s = m.particle_states()[1]
    s.position[0] = 30.0
    assert lib.lbm_set_particle(m.handle, 2, C.byref(s)) == 0
    assert _launches(lib, m, 30) == 1


@pytest.mark.parametrize("n,parts,walls,storage,resident", [
    ((64, 64), [], False, "f32", True), ((64, 64), [], False, "f64", False), ((87, 87), [], False, "f64", False),
    ((400, 400), [], True, "f32", True), ((440, 440), [], True, "f32", False), ((441, 440), [], True, "f32", True),
    ((440, 440), [], True, "f64", True), ((600, 600), ONE, True, "f32", True), ((700, 700), ONE, True, "f32", False),
    ((701, 700), ONE, True, "f32", True), ((700, 700), ONE, False, "f32", True), ((700, 700), ONE, True, "f64", True)])
def test_grids_on_both_sides_of_the_limits(lib, n, parts, walls, storage, resident):
    """Larger grids, and FP64 fluid alone, are faster in stream order; a first call of some length runs as one launch
    all the same, instead of building the stream schedule's graphs."""
    m = _model(n, parts, walls=walls, storage=storage)
    in_order = 50 * (1 + bool(parts or walls) + bool(parts))
    assert [_launches(lib, m, 50) for _ in range(2)] == [1, 1 if resident else in_order]


@pytest.mark.parametrize("n,radius,parts,walls,least", [
    ((64, 64), 6.0, 0, False, 10), ((61, 40), 6.0, 0, True, 3), ((257, 256), 6.0, 0, True, 10),
    ((64, 64), 6.0, 1, False, 2), ((128, 96), 6.8, 1, False, 3), ((201, 65), 6.0, 1, True, 2),
    ((200, 160), 26.0, 1, False, 3), ((200, 160), 27.0, 1, False, 5), ((120, 90), 6.0, 2, False, 5),
    ((520, 510), 6.0, 2, False, 10)])
def test_short_calls_run_in_stream_order(lib, n, radius, parts, walls, least):
    """A launch of many ticks costs more than a graph replay, so calls of few ticks do not take it."""
    import lbmengine as lbm
    m = _model(n, [], walls=walls)
    for k in range(parts):
        lbm.addSquirmer(m, radius=radius, position=[0.3 + 40.0 * k, 0.2], massDensity=3.0, swimmingSpeed=1e-3, beta=2.0,
                        swimmingDirection=[0.8, 0.6], coupleForces=True, coupleTorques=True)
    per_tick = 1 + bool(parts or walls) + bool(parts)
    for _ in range(2):
        assert _launches(lib, m, least - 1) == (least - 1) * per_tick
        assert _launches(lib, m, least) == 1
