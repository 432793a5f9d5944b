"""Galerkin products A_c = R A P on both sides of the row kernels' limits: a warp per row below 192
(A entry, R entry) pairs and 128 columns, a block per row above, where a row's pairs and products are
cut into runs of 256 and 1,024.  Coarse operators are bit-identical to the oracle's (entry order, values)."""
import numpy as np
import pytest

import oracle
from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,phases,channels", [((7, 5, 3), 2, 0),  # few rows, all short
                                                  ((17, 13, 9), 3, 4),  # runs end inside rows
                                                  ((23, 61, 13), 2, 6),  # rows of thousands of pairs
                                                  ((64, 3, 65), 2, 0)])  # thin: long rows on few columns
def test_coarse_operators_bit_exact(grid, phases, channels):
    s = synth.reservoir_system(*grid, 5, phases=phases, channelised_layers=channels)
    a, _ = oracle.bsr_decouple(s.ia, s.ja, s.a, s.block_size, s.b, 1)
    G = CprGmres(decouple=1).setup(s.ia, s.ja, s.a, s.block_size)
    O = oracle.OracleCPR(s.ia, s.ja, a, s.block_size)
    assert G.num_levels() == O.num_levels()
    for lev in range(1, O.num_levels()):
        for u, v in zip(G.level_matrix(lev, 0)[:3], O.level_matrix(lev, 0)[:3]):
            assert np.array_equal(u, v), f"A{lev}"
