"""Boundary layouts of the ring table's range, for the CPU and the GPU tests:
every kind of field it accepts on every face, split faces, AxisLF segments in
each position, and (REFUSED) layouts only the general path runs."""
from __future__ import annotations

import dataclasses

from tests import cases

segment = cases.segment
WALL = dict(v_r=("expr", "v_z * r_z"), H_r=("expr", "H_z * r_z"))
AXIS = dict(rho="axis_lf", v_z="axis_lf", e="axis_lf", H_z="axis_lf", v_r=("dirichlet", 0.0),
            v_phi=("dirichlet", 0.0), H_r=("dirichlet", 0.0), H_phi=("dirichlet", 0.0))


def channel(L, M):
    return cases.channel_config(L=L, M=M, a=0.12, amp=1.3, beta=0.3)


def thruster(L, M):
    """The thruster's three inner-wall segments, contiguous at any L."""
    cfg = cases.reference_default_config(L=L, M=M)
    a = int(235 * L / 800)
    b = max(a + 1, int(263 * L / 800))
    s = cfg.bc_m_lo.segments
    s[0].global_hi, s[1].global_lo, s[1].global_hi, s[2].global_lo = a, a + 1, b, b + 1
    return cfg


def split(L, M):
    """Faces of several segments, overlaps included (the last one decides), every
    operation and geometry symbol."""
    cfg = channel(L, M)
    h = M // 2
    cfg.bc_l_lo.segments = [
        segment((0, h), rho=("dirichlet", 1.0), v_z=("neumann", 0.01), e=("expr", "beta + r"),
                H_phi=("expr", "2 * 0.2 / r")),
        segment((h, -1), rho=("expr", "1.2 - dr"), v_z=("dirichlet", 0.1),
                v_phi=("expr", "z - 0.01"), H_phi=("expr", "H_phi_nb * r_nb"))]
    cfg.bc_l_hi.segments = [segment((0, h), e=("neumann", 0.001)), segment((h + 1, -1),
                                                                         v_r=("expr", "v_z * r_z"))]
    cfg.bc_m_hi.segments = [segment(v_r=("expr", "v_z_nb * r_z_nb")),
                            segment((L // 2, -1), **WALL)]
    cfg.bc_m_lo.segments = [segment(**WALL), segment((1, L // 3), H_z=("neumann", 0.001),
                                                     v_r=("expr", "v_z * r_z"))]
    cfg.init()
    return cfg


def axis_everywhere(L, M):
    cfg = channel(L, M)
    cfg.bc_m_lo.segments = [segment(**AXIS)]
    cfg.init()
    return cfg


def axis_mixed(L, M):
    """AxisLF next to constants and walls: rows whose half-stencil reads the new
    value of the row before them."""
    cfg = channel(L, M)
    a, b = L // 3, 2 * L // 3
    cfg.bc_m_lo.segments = [
        segment((0, a), **WALL),
        segment((a + 1, b), **{**AXIS, "v_z": ("dirichlet", 0.15), "H_z": ("expr", "H_z0 * 0")}),
        segment((b + 1, -1), **AXIS)]
    cfg.init()
    return cfg


ACCEPTED = [channel, thruster, split, axis_everywhere, axis_mixed]


def uncovered(L, M):
    cfg = channel(L, M)
    cfg.bc_m_hi.segments = [segment((2, -1), **WALL)]
    cfg.init()
    return cfg


def interpreted(L, M):
    cfg = channel(L, M)
    cfg.bc_l_lo.segments = [segment(rho=("expr", "1 + 0.1 * sin(pi * r)"), v_z=("dirichlet", 0.1))]
    cfg.init()
    return cfg


def axis_overlap(L, M):
    cfg = channel(L, M)
    cfg.bc_m_lo.segments = [segment(**WALL), segment((L // 2, -1), **AXIS)]
    cfg.init()
    return cfg


def axis_unordered(L, M):
    cfg = channel(L, M)
    cfg.bc_m_lo.segments = [segment((L // 2, -1), **WALL), segment((0, L // 2 - 1), **AXIS)]
    cfg.init()
    return cfg


def axis_free_vz(L, M):
    cfg = channel(L, M)
    cfg.bc_m_lo.segments = [segment(**{**AXIS, "v_z": "neumann"})]
    cfg.init()
    return cfg


REFUSED = [uncovered, interpreted, axis_overlap, axis_unordered, axis_free_vz]
