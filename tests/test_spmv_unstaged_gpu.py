"""The unstaged SpMV kernels at their edges, bit-exact against the oracle: arrays that start off 16-byte
boundaries, empty rows, a last block with few rows.  2x2 FP64 blocks run the slab kernel, which copies the range
of 128 rows to shared memory (its ends value by value off a boundary), unless it holds more than 1,024 blocks:
"fits" and "exceeds" are the two sides.  3x3 blocks and FP32 values run the direct kernel, one thread per
component, on rows of the same kinds."""
import numpy as np
import pytest

import oracle
from jxpamg_all_b200 import lib

pytestmark = pytest.mark.gpu

# bs 2: the slab kernel's rows per block of threads and the blocks its shared memory holds; bs 3: as many rows
# of seven blocks
ROWS, CAP = {2: 128, 3: 64}, {2: 1024, 3: 448}


def pattern(bs, lens, seed):
    nb = len(lens)
    rng = np.random.default_rng(seed)
    ia = np.zeros(nb + 1, np.int32)
    ia[1:] = np.cumsum(lens)
    ja = rng.integers(0, nb, ia[-1]).astype(np.int32)
    return ia, ja, rng.standard_normal(len(ja) * bs * bs), rng.standard_normal(nb * bs)


def lengths(kind, bs):
    rows, cap = ROWS[bs], CAP[bs]
    if kind == "ragged":  # empty and short rows, a last block of one row
        return [(3 * i) % 9 for i in range(2 * rows + 1)]
    total = cap if kind == "fits" else cap + 1
    q, r = divmod(total, rows)
    return [q + (i < r) for i in range(rows)] + [2] * 5


@pytest.mark.parametrize("bs", [2, 3])
@pytest.mark.parametrize("kind", ["ragged", "fits", "exceeds"])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("off_a,off_j", [(0, 0), (1, 3), (2, 1), (3, 2)])
def test_unstaged_spmv_bit_exact(bs, kind, f32, off_a, off_j):
    from gpu_util import dev, host, ptr, stream

    ia, ja, a, x = pattern(bs, lengths(kind, bs), 7)
    a = a.astype(np.float32) if f32 else a
    ad, jd = dev(np.concatenate([np.zeros(off_a, a.dtype), a])), dev(np.concatenate([np.zeros(off_j, np.int32), ja]))
    iad, xd, yd = dev(ia), dev(x), dev(np.zeros_like(x))
    so = lib.load()
    fn = so.jxcpr_bsr_matvec_dev_f32 if f32 else so.jxcpr_bsr_matvec_dev
    lib.check(fn(len(ia) - 1, bs, len(ja), ptr(iad), ptr(jd) + 4 * off_j, ptr(ad) + a.itemsize * off_a, 1.0, ptr(xd),
                 0.0, ptr(yd), 0, stream()))
    assert np.array_equal(host(yd), oracle.bsr_matvec(ia, ja, a.astype(np.float64), bs, x))
