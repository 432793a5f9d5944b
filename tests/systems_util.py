"""Systems with long or many-entried rows, built from the synthetic ones."""
import numpy as np


def with_wells(s, wells, connections, seed):
    """The system with `wells` further block rows, each coupled both ways to `connections` random cells."""
    rng = np.random.default_rng(seed)
    nb, bs = s.num_block_rows, s.block_size
    a = s.a.reshape(-1, bs, bs).copy()
    rows, cols, vals = [np.repeat(np.arange(nb), np.diff(s.ia))], [s.ja], [a]
    for w in range(nb, nb + wells):
        cells = np.sort(rng.permutation(nb)[:connections])
        t = rng.uniform(0.1, 2.1, connections)
        a[s.ia[cells], 0, 0] += t  # the diagonal block is a row's first
        off, diag = np.zeros((connections, bs, bs)), np.eye(bs)[None].copy()
        off[:, 0, 0], diag[0, 0, 0] = -t, 1.001 * t.sum()
        rows += [[w], np.full(connections, w), cells]
        cols += [[w], cells, np.full(connections, w)]
        vals += [diag, off, off]
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((cols, rows != cols, rows))
    ia = np.zeros(nb + wells + 1, np.int32)
    ia[1:] = np.cumsum(np.bincount(rows))
    return ia, cols[order].astype(np.int32), vals[order].reshape(-1), bs


def random_graph(n, neighbours, seed):
    """2x2 blocks on a random graph of about `neighbours` neighbours a row, the pressure part an M-matrix."""
    rng = np.random.default_rng(seed)
    cols = [set() for _ in range(n)]
    for i in range(n):
        for j in rng.integers(0, n, neighbours // 2):
            if j != i:
                cols[i].add(int(j))
                cols[int(j)].add(i)
    ia, ja = [0], []
    for i in range(n):
        ja += [i] + sorted(cols[i])
        ia.append(len(ja))
    ia, ja = np.array(ia, np.int32), np.array(ja, np.int32)
    a = np.zeros((len(ja), 2, 2))
    a[:, 0, 0] = -rng.uniform(0.1, 1.0, len(ja))
    a[ia[:-1], 0, 0] = 0.0
    a[ia[:-1], 0, 0] = -1.01 * np.add.reduceat(a[:, 0, 0], ia[:-1])
    a[ia[:-1], 1, 1] = 1.0
    return ia, ja, a.reshape(-1), 2
