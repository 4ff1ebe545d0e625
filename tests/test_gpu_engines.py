"""One solver through several engines: the one-kernel steps of a graph run or of
Advance, the persistent loop, a batch and the two-kernel form, each starting from
what the one before it left.  Every plane, t, dt and wave speed must be those of
a solver that took the two-kernel form throughout (its boundary kernel leaves
the wall lines after every step)."""
import numpy as np
import pytest

from tests import cases, ring_layouts

pytestmark = pytest.mark.gpu

LAYOUTS = [ring_layouts.thruster, ring_layouts.axis_mixed, ring_layouts.axis_everywhere,
           ring_layouts.channel, ring_layouts.split]


class Walk:
    """A solver and the reference beside it, the same steps in both."""

    def __init__(self, pkg, cfg):
        case = cases.make_case(cfg)
        self.pkg, self.dt = pkg, 1e-6
        self.a = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast")
        self.ref = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast")
        self.ref.ring_overlap = True
        self.batch = pkg.BatchSolver([self.a])

    def _run(self, s, n, **kw):
        return s.run(T=1e300, dt=self.dt, adaptive=True, max_steps=n, steps_per_graph=10, **kw)

    def go(self, how, n):
        want = None
        if how == "advance":
            for _ in range(n):
                self.a.Advance(self.dt)
                self.ref.Advance(self.dt)
                dt = self.a.ComputeDt(self.dt)
                assert dt == self.ref.ComputeDt(self.dt)
                assert self.a.MaxWaveSpeed() == self.ref.MaxWaveSpeed()
                self.dt = dt
        else:
            if how == "batch":
                got = self.batch.run(self.pkg.BatchPlan([2], [0]), T=1e300, dt=self.dt,
                                     adaptive=True, max_steps=n).runs[0]
            elif how == "two kernels":
                self.a.ring_overlap = True
                got = self._run(self.a, n)
                self.a.ring_overlap = False
            else:
                got = self._run(self.a, n, engine=how)
            want = self._run(self.ref, n)
            assert (got.steps, got.t, got.dt, got.max_wave_speed, got.residual) == \
                (want.steps, want.t, want.dt, want.max_wave_speed, want.residual), (how, n)
            self.dt = want.dt
        np.testing.assert_array_equal(self.a.conserved(), self.ref.conserved(), err_msg=how)

    def close(self):
        self.batch.close()
        self.a.close()
        self.ref.close()


@pytest.mark.parametrize("make", LAYOUTS, ids=lambda f: f.__name__)
@pytest.mark.parametrize("lead", [3, 4])
@pytest.mark.parametrize("whole", ["graph", "advance"])
@pytest.mark.parametrize("other", ["persistent", "batch", "two kernels"])
def test_boundary_after_whole_steps(pkg, make, lead, whole, other):
    """The faces' old wall values, after an odd and an even number of whole steps."""
    w = Walk(pkg, make(40, 31))
    w.go(whole, lead)
    w.go(other, 5)
    w.close()


@pytest.mark.parametrize("lead", [2, 3, 4])
@pytest.mark.parametrize("between", [1, 2, 3])
@pytest.mark.parametrize("other", ["persistent", "batch", "two kernels"])
def test_wave_speed_of_whole_steps_after_others(pkg, lead, between, other):
    """The thruster's start-up, its wave speed falling every few steps: a maximum
    left from before the other engine's steps would show in the next one's."""
    w = Walk(pkg, ring_layouts.thruster(40, 31))
    speeds = []
    for how, n in (("graph", lead), (other, between), ("graph", 1), ("advance", 2),
                   (other, between), ("advance", 1), (other, between), ("graph", 12)):
        w.go(how, n)
        speeds.append(w.ref.MaxWaveSpeed())
    assert all(b < a for a, b in zip(speeds, speeds[1:])), speeds
    assert w.a.MaxWaveSpeed() == speeds[-1]
    w.close()


def test_continued_runs_reuse_their_graphs(pkg):
    """Runs from odd and from even steps need a graph each, whatever the number of
    them and the new initial states, monitored ones one more; with a change check
    there is one for each offset too, the last 16 kept."""
    case = cases.make_case(ring_layouts.channel(40, 31))
    a = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast", with_prev=True)
    b = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="fast", with_prev=True)
    b.ring_overlap = True

    def both(**kw):
        r = [s.run(T=1e300, dt=1e-6, adaptive=True, **kw) for s in (a, b)]
        assert (r[0].steps, r[0].t, r[0].dt, r[0].change) == \
            (r[1].steps, r[1].t, r[1].dt, r[1].change)
        np.testing.assert_array_equal(a.conserved(), b.conserved())

    for n in (100, 100, 31, 100, 7, 100):
        both(max_steps=n, steps_per_graph=10)
    a.run(T=1e300, dt=1e-6, max_steps=33, steps_per_graph=10, monitor=lambda rep: None,
          monitor_every=20)
    b.run(T=1e300, dt=1e-6, max_steps=33, steps_per_graph=10)
    a.set_physical(case.phys)
    b.set_physical(case.phys)
    both(max_steps=100, steps_per_graph=10)
    assert a.graph_builds() == 3
    check = dict(steps_per_graph=20, convergence_threshold=1e-30, check_frequency=20)
    for n in (60, 60, 47, 60, 13, 60, 60):   # two offsets, their parities with them
        both(max_steps=n, **check)
    assert a.graph_builds() == 5
    for _ in range(40):                      # all 20 offsets, twice
        both(max_steps=21, **check)
    a.close()
    b.close()
