"""One-kernel fast steps (lf_step_kernel) against the two-kernel form with the
ring recomputed by the general path (ring_overlap): every plane, dt, t and wave
speed bit for bit, over the layouts the ring table accepts, at sizes around the
strips' and bands' edges, through the graph loop, the per-call loop, an
odd number of steps per graph, a monitored run and the relative-change check."""
import numpy as np
import pytest

from tests import cases, ring_layouts

pytestmark = pytest.mark.gpu


def _two(pkg, cfg, **kw):
    case = cases.make_case(cfg)
    a = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast", **kw)
    b = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast", **kw)
    b.ring_overlap = True
    return a, b


def _same(a, b):
    np.testing.assert_array_equal(a.conserved(), b.conserved())


@pytest.mark.parametrize("make", ring_layouts.ACCEPTED, ids=lambda f: f.__name__)
@pytest.mark.parametrize("L,M", [(4, 3), (7, 30), (33, 31), (40, 60), (61, 61)])
def test_layouts_and_sizes_bitwise(pkg, make, L, M):
    a, b = _two(pkg, make(L, M))
    dt = 1e-6
    for n, per in ((60, 20), (31, 31)):
        x = a.run(T=1e300, dt=dt, adaptive=True, max_steps=n, steps_per_graph=per)
        y = b.run(T=1e300, dt=dt, adaptive=True, max_steps=n, steps_per_graph=per)
        assert (x.steps, x.t, x.dt, x.max_wave_speed, x.residual) == \
            (y.steps, y.t, y.dt, y.max_wave_speed, y.residual)
        _same(a, b)
        dt = x.dt
    a.close()
    b.close()


@pytest.mark.parametrize("L,M", [(1300, 640), (2600, 1100)])
def test_large_grids_share_warps_between_ring_and_bands(pkg, L, M):
    """Bands of more than a few rows: ring warps with (shorter) bands, spread over
    the blocks or, for a state far larger than L2, in task order."""
    a, b = _two(pkg, ring_layouts.channel(L, M))
    x = a.run(T=1e300, dt=1e-6, adaptive=True, max_steps=21)
    y = b.run(T=1e300, dt=1e-6, adaptive=True, max_steps=21)
    assert (x.t, x.dt, x.max_wave_speed) == (y.t, y.dt, y.max_wave_speed)
    _same(a, b)
    a.close()
    b.close()


def test_fixed_dt_per_call_switching_and_end_time(pkg):
    a, b = _two(pkg, ring_layouts.thruster(60, 33))
    for _ in range(7):
        a.Advance(1e-6)
        b.Advance(1e-6)
        assert a.ComputeDt(1e-6) == b.ComputeDt(1e-6)
    _same(a, b)
    a.ring_overlap = True      # from whole steps to the two-kernel form ..
    b.ring_overlap = False     # .. and the other way
    for s in (a, b):
        r = s.run(T=s.time()[0] + 1e-5, dt=1e-6, adaptive=False, max_steps=1000,
                  steps_per_graph=3)
        assert r.steps == 10
    assert a.time() == b.time()
    _same(a, b)
    a.close()
    b.close()


def test_monitor_residual_and_change_checks(pkg):
    cfg = ring_layouts.channel(48, 24)
    a, b = _two(pkg, cfg, with_prev=True)
    got = []
    for s in (a, b):
        recs = []
        r = s.run(T=1e300, dt=1e-5, max_steps=230, residual_every=10, monitor=recs.append,
                  monitor_every=70)
        got.append((r.steps, r.t, r.residual, [(m.step, m.t, m.dt, m.max_wave_speed) for m in recs]))
    assert got[0] == got[1] and [m[0] for m in got[0][3]] == [70, 140, 210]
    got = []
    for s in (a, b):
        r = s.run(T=1e300, dt=1e-5, max_steps=300, convergence_threshold=1e-30,
                  check_frequency=30, steps_per_graph=60)
        got.append((r.steps, r.t, r.change, r.converged))
        r = s.run(T=1e300, dt=1e-5, max_steps=300, convergence_threshold=10.0,
                  check_frequency=7)   # met at the first check: a step count divisible by 7
        got[-1] += (r.steps, r.t, r.change, r.converged)
        assert r.converged and (230 + 300 + r.steps) % 7 == 0
    assert got[0] == got[1]
    _same(a, b)
    a.close()
    b.close()
