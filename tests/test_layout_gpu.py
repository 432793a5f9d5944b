"""The operators' layouts chosen by size (sliced ELL with 1 to 32 lanes per row, CSR) against the layouts
without autotuning: one FP64 V-cycle agrees to rounding.  The grids and thresholds give levels of 300 to
60,000 rows with 5 to 150 entries."""
import numpy as np
import pytest

from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,phases,theta", [((9, 8, 7), 2, 0.25), ((37, 41, 23), 2, 0.25), ((37, 41, 23), 2, 0.7),
                                               ((30, 33, 61), 2, 0.25), ((21, 34, 19), 3, 0.5)])
@pytest.mark.parametrize("smoother", [0, 1])
def test_layouts_agree(grid, phases, theta, smoother):
    s = synth.reservoir_system(*grid, 9, phases=phases)
    rp = np.random.default_rng(2).standard_normal(s.num_block_rows)
    out = []
    for autotune in (0, 1):
        G = CprGmres(decouple=1, smoother_order=1, coarse_exact=0, precision=0, fast_smoother=smoother,
                     strong_threshold=theta, autotune=autotune).setup(s.ia, s.ja, s.a, s.block_size)
        out.append(G.vcycle(rp))
        G.close()
    # sums of at most a few hundred products in another order, a handful of levels and passes
    assert np.linalg.norm(out[0] - out[1]) <= 1e-12 * np.linalg.norm(out[0])
