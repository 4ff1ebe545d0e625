"""The exact interior kernel's shared-memory tiles (32 x 8 cells and their halo)
at sizes around the tile's edges: bit for bit the oracle, first step included."""
import numpy as np
import pytest

from oracle import bind
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,M", [(4, 3), (7, 32), (8, 33), (9, 34), (16, 65), (17, 66)])
def test_exact_steps_bitwise_at_tile_edges(pkg, L, M):
    case = cases.make_case(cases.channel_config(L=L, M=M, a=0.1, amp=1.4))
    s = pkg.GpuSolver(case.cfg, case.grid, case.phys, precision="exact")
    oracle = bind.Port(case.oracle_dict())
    dt = 1e-4
    for _ in range(6):
        s.Advance(dt)
        oracle.advance(dt)
        np.testing.assert_array_equal(s.conserved(), oracle.conserved())
        assert s.MaxWaveSpeed() == oracle.max_wave_speed()
    s.close()
