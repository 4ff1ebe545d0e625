"""The ring evaluated from the ring table and the step's input state alone
(lf_step_kernel's ring warps), on the CPU, against the general boundary path
(bc_ring_final) over every kind of layout the table accepts; and what it
refuses."""
import numpy as np
import pytest

from oracle import bind
from tests import cases, ring_layouts
from tests.emu import Emu


def _has_ring(emu):
    return bool(emu.lib.mpd_emu_has_ring(emu.h))


@pytest.mark.parametrize("L,M", [(4, 3), (5, 4), (12, 9), (40, 31)])
@pytest.mark.parametrize("make", ring_layouts.ACCEPTED, ids=lambda f: f.__name__)
def test_table_ring_is_the_general_ring_bitwise(make, L, M):
    cfg = make(L, M)
    case = cases.make_case(cfg)
    a, b = Emu(case, "fast"), Emu(case, "fast")
    assert _has_ring(a)
    for _ in range(4):
        a.advance(1e-6)
        b.advance(1e-6, order=3)
        np.testing.assert_array_equal(b.conserved(), a.conserved())


@pytest.mark.parametrize("make", ring_layouts.REFUSED, ids=lambda f: f.__name__)
def test_refused_layouts_keep_the_general_path(make):
    emu = Emu(cases.make_case(make(12, 9)), "fast")
    assert not _has_ring(emu)


def test_constant_parts_of_an_expression_fold_to_the_interpreters_bits():
    """amp * 0.2 / r: the constant product meets first, as in the sweep."""
    for expr in ("1.3 * 0.2 / r", "(beta + 0.1) * r", "-2 * r", "r / (3 * 0.7)"):
        cfg = ring_layouts.channel(12, 9)
        cfg.bc_l_lo.segments[0].H_phi = cases.pkg.FieldCond("expression", 0.0, expr)
        case = cases.make_case(cfg)
        a, b = Emu(case, "fast"), Emu(case, "fast")
        assert _has_ring(a)
        oracle = bind.Port(case.oracle_dict())
        exact = Emu(case, "exact")
        for _ in range(3):
            a.advance(1e-5)
            b.advance(1e-5, order=3)
            exact.advance(1e-5)
            oracle.advance(1e-5)
            np.testing.assert_array_equal(b.conserved(), a.conserved())
            np.testing.assert_array_equal(exact.conserved(), oracle.conserved())


@pytest.mark.parametrize("L,M", [(5, 4), (40, 31)])
@pytest.mark.parametrize("make", ring_layouts.ACCEPTED, ids=lambda f: f.__name__)
def test_general_ring_after_table_rings_bitwise(make, L, M):
    """The general path starts from the walls' old values, which table rings
    leave behind: they come from the state then, for either step parity."""
    case = cases.make_case(make(L, M))
    a, b = Emu(case, "fast"), Emu(case, "fast")
    for order in (0, 3, 0, 3, 3, 0, 0, 3, 3, 3, 0):
        a.advance(1e-5)
        b.advance(1e-5, order=order)
        np.testing.assert_array_equal(b.conserved(), a.conserved())


@pytest.mark.parametrize("make", ring_layouts.ACCEPTED, ids=lambda f: f.__name__)
def test_indexes_of_the_table_are_checked_on_the_host(make):
    """The device takes them unchecked: every table in range, none with an index
    past its end."""
    L, M = 12, 9
    emu = Emu(cases.make_case(make(L, M)), "fast")
    ok = lambda *a: bool(emu.lib.mpd_emu_ring_in_range(emu.h, *a))
    length, cfg = max(L + 2, M + 3), make(L, M)
    nseg = sum(len(f.segments) for f in (cfg.bc_l_lo, cfg.bc_l_hi, cfg.bc_m_lo, cfg.bc_m_hi))
    assert ok(-1, 0, 0)
    for face, (lo, hi) in enumerate([(1, M), (1, M + 1), (2, L - 1), (1, L - 1)]):
        for k in (lo, hi):
            assert ok(0, face * length + k, nseg - 1) and not ok(0, face * length + k, nseg)
    assert not ok(1, 0, 9) and not ok(1, 0, -1)
    assert any(not ok(2, s, 8) and not ok(2, s, -1) and not ok(3, s, 22) and not ok(4, s, -2)
               for s in range(nseg))
