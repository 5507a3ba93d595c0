"""The device memory an LP is admitted with (pdlp_estimate_device_bytes) covers
what its upload and solve hold at once, where non-zeros, rows or columns make up
most of it, in each precision; and an upload needs no more than the solve."""
import ctypes as C

import numpy as np
import pytest

import cupdlpx as cp
from test_gpu_fp32_sums import matrix
from test_gpu_solve import params

pytestmark = pytest.mark.gpu

SHAPES = {
    "non_zeros": ([130] * 40000, 40000),        # all rows in the front, on both sides
    "non_zeros_in_strips": ([40] * 120000, 130000),
    "columns": ([3] * 20000, 1500000),
    "rows": ([1] * 1500000, 20000),
    "several_lanes": ([9] * 3000, 4000),
    "team": ([8] * 100000, 150000),
}


@pytest.mark.parametrize("precision", [cp.PRECISION_FP64, cp.PRECISION_FP32_REFINE,
                                       cp.PRECISION_FP32_MATRIX])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_estimate_covers_upload_and_solve(lib, oracle, name, precision):
    lengths, n = SHAPES[name]
    prob, (ptr, _, _), _, _ = matrix(lengths, n, 41)
    prob.set_start(np.zeros(n), np.zeros(len(lengths)))
    lib.pdlp_pooled_memory_high.restype = C.c_longlong
    p = params(oracle, eps=1e-14, iteration_limit=30)
    lib.pdlp_pooled_memory_high(1)
    dp = cp.DeviceProblem(prob)
    upload = lib.pdlp_pooled_memory_high(0)
    dp.free()
    lib.pdlp_pooled_memory_high(1)
    cp.solve(prob, p, precision=precision)
    high = lib.pdlp_pooled_memory_high(0)
    nnz = int(ptr[-1])
    estimate = lib.pdlp_estimate_device_bytes(len(lengths), n, nnz, precision)
    assert 0 < high <= estimate
    assert upload <= high
