"""Sliced ELL operators with 16-bit columns (distances from the row; at least 2^22 stored entries).

Coarse levels: bit for bit the 32-bit columns' V-cycle (the cooperative tail kernel, which never takes level 0,
reads the 32-bit ones; autotune 0: both runs take the same layouts).

Level 0: against the same operator in CSR, to rounding, and the setup report says which columns it has.  The
layouts come from a tuning file (JXCPR_TUNE_CACHE, read once per process: a child process per layout).  Planes of
32,767 rows are the widest that 16 bits hold in both directions; with planes of 32,768 the next plane is one
too far and level 0 keeps 32-bit columns."""
import os
import subprocess
import sys

import numpy as np
import pytest

from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres

pytestmark = pytest.mark.gpu

EDGES = {(217, 151, 20): True, (256, 128, 20): False}  # grid: 16-bit columns on level 0


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


def edge_vcycles(path):
    """In a child process: the V-cycles of every edge grid, FP64 and FP32, and what the report says of A0."""
    out = {}
    for g, grid in enumerate(EDGES):
        s = synth.reservoir_system(*grid, 9, phases=2)
        rp = np.random.default_rng(2).standard_normal(s.num_block_rows)
        for precision in (0, 1):
            G = CprGmres(decouple=1, smoother_order=1, coarse_exact=0, precision=precision, flexible=precision,
                         fast_smoother=precision).setup(s.ia, s.ja, s.a, s.block_size)
            out[f"v{g}{precision}"] = G.vcycle(rp)
            out[f"r{g}{precision}"] = next(l for l in G.setup_report().splitlines() if "tuned A0 " in l)
            G.close()
    np.savez(path, **out)


def test_near_columns_of_level_0_against_csr(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = []
    for name, sell, lanes in (("sell", 1, 1), ("csr", 0, 2)):
        with open(tmp_path / f"{name}.txt", "w") as f:  # key: operator, rows, entries, value kind, block entries
            for nx, ny, nz in EDGES:
                n = nx * ny * nz
                nnz = 7 * n - 2 * (nx * ny + ny * nz + nz * nx)
                for kind in (0, 1):
                    f.write(f"A0/{n}/{nnz}/{kind}/1 {sell} {lanes} 1.0\n")
        env = dict(os.environ, JXCPR_TUNE_CACHE=str(tmp_path / f"{name}.txt"))
        env["PYTHONPATH"] = os.pathsep.join([root, os.path.join(root, "tests")])
        code = f"import test_near_columns_gpu as t; t.edge_vcycles({str(tmp_path / name)!r})"
        subprocess.run([sys.executable, "-c", code], env=env, check=True, timeout=600)
        res.append(np.load(tmp_path / f"{name}.npz"))
    a, b = res
    for g, near in enumerate(EDGES.values()):
        for precision in (0, 1):
            assert ("16-bit columns" in str(a[f"r{g}{precision}"])) == near, a[f"r{g}{precision}"]
            assert "layout sell" in str(a[f"r{g}{precision}"]) and "layout csr/2" in str(b[f"r{g}{precision}"])
            d = a[f"v{g}{precision}"] - b[f"v{g}{precision}"]
            # 1e-16 / 6e-8 times the 1e5 by which the nearly constant vector comes back (the Jacobian's rows sum
            # to the compressibility); a wrong column is an error of order 1 in every row
            tol = 1e-10 if precision == 0 else 2e-2
            assert np.linalg.norm(d) <= tol * np.linalg.norm(a[f"v{g}{precision}"])
