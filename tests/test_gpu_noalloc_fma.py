"""pdlp_spmv_noalloc adds its products unrounded: in a run of eight consecutive
non-zeros, -fl(ab) and then a b meet in one chain of FMAs, whose result is the
rounding error of fl(ab), exactly.  Rows summed by a thread and by a warp, zeros
elsewhere; and arrays off 16-byte boundaries, which take scalar loads."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# entries of a row, places of the two entries (rows of a multiple of 8 entries
# start with a run; the others' runs start anywhere, so the two are neighbours
# and a row in which a run parts them is left out)
ROWS = {"pair": (2, 0, 1), "eight": (8, 0, 7), "thread": (512, 504, 511),
        "warp": (1024, 840, 847), "odd": (65, 3, 4)}


@pytest.mark.parametrize("name", sorted(ROWS))
@pytest.mark.parametrize("shift", [0, 1])
def test_products_are_not_rounded(lib, name, shift):
    lib.pdlp_spmv_noalloc.restype = C.c_int
    lib.pdlp_spmv_noalloc.argtypes = [C.c_int] * 3 + [C.c_void_p] * 6
    n, first, second = ROWS[name]
    rows = min(31, 2048 // n)  # one tile: no row crosses its end
    rng = np.random.default_rng(n)
    a, b = rng.random(rows) + 1.0, rng.random(rows) + 1.0
    ptr = np.arange(rows + 1, dtype=np.int32) * n
    col = np.full(rows * n, rows, dtype=np.int32)
    val = np.zeros(rows * n)
    for r in range(rows):
        val[r * n + first], col[r * n + first] = -(a[r] * b[r]), rows
        val[r * n + second], col[r * n + second] = a[r], r
    x = np.append(b, 1.0)
    exact = [float(Fraction(a[r]) * Fraction(b[r]) - Fraction(a[r] * b[r])) for r in range(rows)]
    apart = [(r * n + first) // 8 != (r * n + second) // 8 for r in range(rows)]
    exact = [0.0 if p else e for p, e in zip(apart, exact)]
    assert np.count_nonzero(exact) > 0
    dev = torch.device("cuda:0")
    # columns and values `shift` entries past the start of their allocations
    d = [torch.from_numpy(np.concatenate([np.zeros(k, v.dtype), v])).to(dev)[k:]
         for v, k in ((ptr, 0), (col, shift), (val, shift), (x, 0))]
    y = torch.zeros(rows, dtype=torch.float64, device=dev)
    torch.cuda.synchronize(dev)
    assert lib.pdlp_spmv_noalloc(rows, rows + 1, rows * n, *(t.data_ptr() for t in d),
                                 y.data_ptr(), None) == 0
    assert y.cpu().tolist() == exact
