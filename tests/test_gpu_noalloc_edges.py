"""pdlp_spmv_noalloc at the edges of its tiles and of its two row paths.

The kernel cuts tiles at every 2,048 non-zeros; a thread adds a row of at most
64 products of a tile, a warp a longer one; a row that crosses tiles is added
from its tiles' partial sums, by a warp when there are more than 32 of them.
"""
import ctypes as C

import numpy as np
import pytest

import cupdlpx as cp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LENGTHS = {
    "one_row_2047": [2047],
    "one_row_2048": [2048],
    "one_row_2049": [2049],
    "rows_end_at_tiles": [2048, 0, 2048, 0, 0],
    "rows_straddle_tiles": [2047, 2, 2046, 3, 1],
    "thread_or_warp_rows": [31, 32, 33, 0, 34] * 40,
    "thread_or_warp_rows_64": [63, 64, 65, 0, 66] * 40,
    "piece_of_32_or_33": [2016, 64, 1999, 50],
    "piece_of_64_or_65": [1984, 128, 1919, 130],
    "32_partials_or_33": [7, 2048 * 33, 5, 2048 * 34, 9],
    "empty_rows_at_ends": [0] * 300 + [1] * 2100 + [0] * 300,
    "no_non_zeros": [0, 0, 0],
}


@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_noalloc_edges_match_oracle(lib, oracle, name):
    lib.pdlp_spmv_noalloc.restype = C.c_int
    lib.pdlp_spmv_noalloc.argtypes = [C.c_int] * 3 + [C.c_void_p] * 6
    rng = np.random.default_rng(len(name))
    lengths = np.array(LENGTHS[name])
    cols = 5000
    ptr = np.zeros(len(lengths) + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(lengths)
    nnz = int(ptr[-1])
    col = rng.integers(0, cols, size=nnz).astype(np.int32)  # entries of a row may repeat
    val, x = rng.standard_normal(nnz), rng.standard_normal(cols)
    y_cpu = np.zeros(len(lengths))
    oracle.oracle_spmv(len(lengths), cp.as_ip(ptr), cp.as_ip(col), cp.as_dp(val), cp.as_dp(x),
                       cp.as_dp(y_cpu), 0)
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(a).to(dev) for a in (ptr, col, val, x)]
    d_y = torch.full((len(lengths),), float("nan"), dtype=torch.float64, device=dev)
    torch.cuda.synchronize(dev)
    rc = lib.pdlp_spmv_noalloc(len(lengths), cols, nnz, *(t.data_ptr() if t.numel() else None
                                                          for t in d), d_y.data_ptr(), None)
    assert rc == 0
    absum = np.zeros(len(lengths))
    np.add.at(absum, np.repeat(np.arange(len(lengths)), lengths), np.abs(val * x[col]))
    # both sums differ from the exact one by at most n u sum|a x|
    assert np.all(np.abs(d_y.cpu().numpy() - y_cpu) <= 2 * 1.2e-16 * np.maximum(lengths, 1) * absum)
