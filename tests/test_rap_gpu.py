"""Galerkin products A_c = R A P on both sides of the row kernels' limits: a warp per row below 192
(A entry, R entry) pairs and 128 columns, a block per row above, where a row's pairs and products are
cut into runs of 256 and 1,024; a row with more than 192 columns in one of eight hash classes goes to a
thread, and the blocks' pass is repeated where their rows have more than 192 columns in the mean.  Coarse
operators are bit-identical to the oracle's (entry order, values)."""
import numpy as np
import pytest

import oracle
from jxpamg_all_b200 import synth
from jxpamg_all_b200.solver import CprGmres
from systems_util import random_graph, with_wells

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


def check(ia, ja, a, bs):
    """The hierarchy bit for bit; returns per coarse level (pairs of each row, R entries, columns)."""
    G = CprGmres(decouple=0).setup(ia, ja, a, bs)
    O = oracle.OracleCPR(ia, ja, a, bs)
    assert G.num_levels() == O.num_levels()
    rows = []
    for lev in range(1, O.num_levels()):
        pia, pja = O.level_matrix(lev - 1, 1)[:2]
        fine = np.diff(O.level_matrix(lev - 1, 0)[0])
        want = O.level_matrix(lev, 0)[:3]
        for u, v in zip(G.level_matrix(lev, 0)[:3], want):
            assert np.array_equal(u, v), f"A{lev}"
        nc = len(want[0]) - 1
        pairs = np.bincount(pja, np.repeat(fine, np.diff(pia)), nc)
        rows.append((pairs, np.bincount(pja, minlength=nc), np.diff(want[0])))
    G.close()
    return rows


def test_rows_beyond_the_block_tables():
    """Wells of 1,500 connections: coarse rows of thousands of columns (eight classes hold 1,536 at most), from
    thousands of fine rows (read 256 at a time)."""
    s = synth.reservoir_system(20, 40, 10, 9)
    pairs, entries, cols = check(*with_wells(s, 2, 1500, 5))[0]
    assert np.any((pairs >= 192) & (cols > 8 * 192) & (entries > 256))


def test_blocks_of_many_columns():
    """A random graph: nearly every coarse row couples to every other, so that the blocks' first room (192
    columns a row) does not suffice though no class overflows, and short rows leave the warp kernel's table."""
    pairs, entries, cols = check(*random_graph(3000, 8, 3))[0]
    block = pairs >= 192
    classes = np.bincount((np.arange(len(cols), dtype=np.uint64) * 2654435761 % 2**32 >> 29).astype(int))
    assert cols[block].mean() > 192 >= classes.max()
    assert np.any(~block & (cols > 128))
