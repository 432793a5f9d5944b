"""Exact-order sweeps from streams in schedule order, bit-identical to the oracle at their edges: a schedule
of a few rows, chunks that split groups, an iterate that fits shared memory and one that stays in global
memory (above 26,000 doubles), 2x2 and 3x3 blocks, the plain update (w = omega = 1)."""
import numpy as np
import pytest

import oracle
from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,phases", [((3, 2, 2), 2), ((14, 9, 21), 2), ((31, 29, 33), 2), ((5, 4, 3), 3),
                                         ((19, 23, 21), 3)])
@pytest.mark.parametrize("w,omega", [(0.7, 0.9), (1.0, 1.0)])
def test_sweeps_bit_exact(grid, phases, w, omega):
    s = synth.reservoir_system(*grid, 3, phases=phases, channelised_layers=grid[2] // 2)
    a, _ = oracle.bsr_decouple(s.ia, s.ja, s.a, s.block_size, s.b, 1)
    G = CprGmres(decouple=1, stage2_relax_weight=w, stage2_omega=omega).setup(s.ia, s.ja, s.a, s.block_size)
    rng = np.random.default_rng(1)
    b, x0 = rng.standard_normal(s.n), rng.standard_normal(s.n)
    assert np.array_equal(G.stage2_sweep(b, x0), oracle.hgs_relax(s.ia, s.ja, a, s.block_size, x0, b, w, omega))
    if (w, omega) == (0.7, 0.9):
        rp = rng.standard_normal(s.num_block_rows)
        O = oracle.OracleCPR(s.ia, s.ja, a, s.block_size)
        assert np.array_equal(G.vcycle(rp), O.vcycle(rp))
