"""The chunk-ordered stage-2 sweep of small colours (a row's whole matrix part read at once, in batches of six
entries) on rows of 1 to 16 blocks, several of them inside the row's own chunk, against the oracle's
restatement in the same order; only the summation order of each row differs."""
import numpy as np
import pytest

import oracle
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu


def system(bs, nb, most, seed):
    rng = np.random.default_rng(seed)
    cols = [set() for _ in range(nb)]
    for i in range(nb):
        for j in rng.integers(max(0, i - 40), min(nb, i + 41), rng.integers(0, most // 2 + 1)):
            if j != i and len(cols[i]) < most - 1 and len(cols[j]) < most - 1:
                cols[i].add(int(j))
                cols[int(j)].add(i)
    ia, ja = [0], []
    for i in range(nb):
        ja += [i] + sorted(cols[i])
        ia.append(len(ja))
    ia, ja = np.array(ia, np.int32), np.array(ja, np.int32)
    a = 0.1 * rng.standard_normal((len(ja), bs, bs)) - 0.2
    a[ia[:-1]] = 4.0 * np.eye(bs) + 0.3 * rng.standard_normal((nb, bs, bs))
    return ia, ja, a.reshape(-1)


@pytest.mark.parametrize("bs", [2, 3])
@pytest.mark.parametrize("most", [7, 8, 13, 16])
@pytest.mark.parametrize("precision", [0, 1])
def test_rows_of_many_lengths(bs, most, precision):
    ia, ja, a = system(bs, 1003, most, 11)
    n = 1003 * bs
    w, om = 0.7, 0.9
    G = CprGmres(decouple=0, smoother_order=1, precision=precision, flexible=precision, stage2_relax_weight=w,
                 stage2_omega=om).setup(ia, ja, a, bs)
    rng = np.random.default_rng(4)
    r, z0 = rng.standard_normal(n), rng.standard_normal(n)
    got = G.stage2_sweep(r, z0)
    G.close()
    want = oracle.hgs_relax_chunked(ia, ja, a, bs, z0, r, 4, w=w, omega=om)
    # FP64 / FP32 rounding of sums of at most 16 block products, diagonal blocks conditioned below two
    assert np.linalg.norm(got - want) <= (1e-12 if precision == 0 else 1e-5) * np.linalg.norm(want)
