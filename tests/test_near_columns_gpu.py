"""Sliced ELL operators with 16-bit columns (distances from the row; at least 2^22 stored entries) give the
32-bit columns' V-cycle bit for bit: the cooperative tail kernel reads the 32-bit ones
(autotune 0: both runs take the same layouts).  A grid whose planes
exceed 32,768 rows keeps 32-bit columns on level 0; one of 32,680 reaches the last representable distances."""
import numpy as np
import pytest

from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(60, 110, 100), (190, 172, 20), (190, 180, 20)])
@pytest.mark.parametrize("precision,smoother", [(0, 0), (1, 1)])
def test_near_columns_bit_exact(grid, precision, smoother):
    s = synth.reservoir_system(*grid, 9, phases=2)
    rp = np.random.default_rng(2).standard_normal(s.num_block_rows)
    out = []
    for tail in (0, 1 << 30):
        G = CprGmres(decouple=1, smoother_order=1, coarse_exact=0, precision=precision, flexible=precision,
                     fast_smoother=smoother, autotune=0, tail_rows=tail).setup(s.ia, s.ja, s.a, s.block_size)
        out.append(G.vcycle(rp))
        G.close()
    assert np.array_equal(out[0], out[1])
