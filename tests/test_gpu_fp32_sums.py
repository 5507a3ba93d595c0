"""FP32 row sums of the default (strip) kernel against those of the fused one.

Below 4,194,304 non-zeros the strip kernel adds a row's products in the fused
kernel's order, whatever the row's place in that kernel's tiles: staged tiles
(segments of 8), the register path (4), rows strided by 2 to 256 lanes and
chunked ones.  Across lanes both add in FP64 and round once to FP32, so the
results are the same bits.

From there on matrices are summed in FP32 pairs (rounded to FP32 once),
but for those with many rows that the pipelined kernel takes at a loss."""
import ctypes as C

import numpy as np
import pytest

import cupdlpx as cp

pytestmark = pytest.mark.gpu


def products(lib, prob, kernel, x, y):
    f = C.POINTER(C.c_float)
    lib.pdlp_gpu_products_fp32.restype = C.c_int
    lib.pdlp_gpu_products_fp32.argtypes = [C.POINTER(cp.LpProblem), C.c_int, f, f, f, f]
    ax, aty = np.zeros(len(y), np.float32), np.zeros(len(x), np.float32)
    assert lib.pdlp_gpu_products_fp32(prob.ptr, kernel, *(a.ctypes.data_as(f)
                                                          for a in (x, y, ax, aty))) == 0
    return ax, aty


def matrix(lengths, n, seed):
    """CSR of random columns; values that FP32 holds exactly."""
    rng = np.random.default_rng(seed)
    lengths = rng.permutation(np.asarray(lengths))
    ptr = np.zeros(len(lengths) + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(lengths)
    col = rng.integers(0, n, ptr[-1]).astype(np.int32)
    val = rng.standard_normal(ptr[-1]).astype(np.float32)
    x = rng.standard_normal(n).astype(np.float32)
    y = rng.standard_normal(len(lengths)).astype(np.float32)
    prob = cp.Problem.from_csr(ptr, col, val.astype(np.float64), n, c=np.zeros(n),
                               lc=np.zeros(len(lengths)), uc=np.ones(len(lengths)),
                               lv=np.zeros(n), uv=np.ones(n))
    return prob, (ptr, col, val), x, y


LENGTHS = {
    # short rows between long ones: tiles whose rows are strided by several
    # lanes, or that hold one short row
    "short_between_long": ([3, 17, 64, 0, 2, 40] * 30 + [300, 450, 90, 65, 512] * 40, 900),
    "short_alone": ([40, 500] * 60, 700),
    "last_tile_one_row": ([16] * 32 + [7], 300),
    "edges": ([63, 64, 65, 0, 1, 31, 32, 33] * 20 + [511, 512, 513, 1023, 1024, 1025, 5000], 6000),
    # rows of 65 to 256 have 32, 16 and 8 lanes
    "wide_32_lanes": ([65, 127, 128, 255, 256, 257, 30] * 20, 9000),
    "wide_16_lanes": ([65, 100, 256, 3] * 600, 9000),
    "wide_8_lanes": ([65, 73, 256, 260, 7] * 1200, 90000),
    # a front in which rows of up to 2,048 are not cut
    "whole_rows": ([2048] * 700 + [2049] * 600 + [1025, 1500, 3000] * 40, 20000),
    "eight_lanes": ([9] * 3000, 5003),
    "four_lanes": ([9] * 9000, 12000),
    "one_lane": ([6] * 45001, 50021),
    # 2M non-zeros or more: tiles of 1,024 and the register path
    "register_path": ([21] * 100000, 300000),
    "register_path_and_long": ([21] * 95000 + [3, 64, 900, 70] * 100, 300000),
}


@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_strip_sums_are_the_fused_kernels(lib, name):
    lengths, n = LENGTHS[name]
    prob, _, x, y = matrix(lengths, n, 29)
    strip, fused = products(lib, prob, -1, x, y), products(lib, prob, 0, x, y)
    assert np.array_equal(strip[0], fused[0])
    assert np.array_equal(strip[1], fused[1])


PAIRS = {
    # one row of 65 entries or more leaves the other rows' sums as they are
    "one_long_row": ([21] * 200000 + [70, 300], 400000),
    "front_of_100": ([100] * 43000, 400000),
    "rows_of_500": ([500] * 8500, 400000),
    # the step kernels of matrices whose rows have at most two entries
    "narrow": ([2, 2, 1, 0, 2] * 1000000, 90000),
}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_large_matrices_are_summed_in_pairs(lib, name):
    lengths, n = PAIRS[name]
    prob, (ptr, col, val), x, y = matrix(lengths, n, 31)
    assert ptr[-1] >= 1 << 22
    ax, aty = products(lib, prob, -1, x, y)
    row = np.repeat(np.arange(len(lengths)), np.diff(ptr))
    for got, to, of, vec in ((ax, row, col, x), (aty, col, row, y)):
        term = val.astype(np.float64) * vec[of]
        exact, size = np.zeros(len(got)), np.zeros(len(got))
        np.add.at(exact, to, term)
        np.add.at(size, to, np.abs(term))
        count = np.bincount(to, minlength=len(got))
        # one rounding to FP32 of the pair; its low part is at most k u size after
        # k products (u = 2^-24) and each of up to four additions to it rounds by
        # u of that
        bar = 2.0 ** -24 * np.abs(exact) + 2.0 * count * (count + 1) * 2.0 ** -48 * size
        assert np.all(np.abs(got - exact) <= bar * (1 + 1e-6))
