"""The operators' layouts chosen by size (sliced ELL with 1 to 32 lanes per row, CSR) against the layouts
without autotuning: one FP64 V-cycle agrees to rounding.  The grids and thresholds give levels of 300 to
60,000 rows with 5 to 150 entries."""
import re

import numpy as np
import pytest

from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres
from systems_util import with_wells

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


@pytest.mark.parametrize("wells,connections", [(0, 0), (2, 50), (3, 900), (1, 9000)])
@pytest.mark.parametrize("precision", [0, 1])
def test_operators_with_long_rows(wells, connections, precision):
    """Operators with a row of more than eight times the mean length take CSR with four times the lanes of the
    mean (1 lane per 4 entries), whatever their number of rows; the others the layout of their size.  The
    V-cycle agrees with the one without autotuning to rounding: in FP64 1e-16 times the 1e5 by which the
    nearly constant vector comes back from these operators, in FP32 (with the constant vector taken out of the
    comparison) 6e-8 times a few hundred."""
    s = synth.reservoir_system(29, 31, 23, 9)
    ia, ja, a, bs = with_wells(s, wells, connections, 5) if wells else (s.ia, s.ja, s.a, s.block_size)
    rp = np.random.default_rng(2).standard_normal(len(ia) - 1)
    out = []
    for autotune in (0, 1):
        G = CprGmres(decouple=0, smoother_order=1, coarse_exact=0, precision=precision, flexible=precision,
                     fast_smoother=precision, autotune=autotune).setup(ia, ja, a, bs)
        out.append(G.vcycle(rp))
        found = re.findall(r"tuned ([APR]\d) rows (\d+) mean ([\d.]+) longest (\d+) layout (\S+)", G.setup_report())
        G.close()
        uneven = 0
        for name, rows, mean, longest, layout in found:
            lanes, mean = 1, float(mean)
            if abs(int(longest) - 8 * max(mean, 1.0)) <= 0.5:
                continue  # the report rounds the mean
            while lanes < 32 and lanes * 4 < mean:
                lanes *= 2
            if int(longest) > 8 * max(mean, 1.0):
                uneven += 1
                assert layout == f"csr/{min(32, 4 * lanes)}", (name, layout)
            elif int(rows) >= 512:
                assert layout.startswith("sell"), (name, layout)
        assert bool(found) == bool(autotune)
        assert not autotune or (uneven > 3 if wells else uneven == 0)
    d = out[0] - out[1]
    if precision:
        d -= d.mean()
    assert np.linalg.norm(d) <= (1e-10 if precision == 0 else 2e-5) * np.linalg.norm(out[0])
