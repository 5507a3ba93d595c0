"""Rows of 65 to 256 entries (wide strips, with 8, 16 or 32 lanes a row) and the
longer ones beside them: points, rescaling and the infinity norm against the CPU
oracle, in matrices that a team runs and in others."""
import numpy as np
import pytest

import cupdlpx as cp
import oracle_lib as ol
from test_gpu_kernels import _gpu_rescale
from test_gpu_solve import params
from test_gpu_strip import _lp

pytestmark = pytest.mark.gpu

# (row lengths, columns, run by a team)
SHAPES = {
    "32_lanes": ([65, 256, 128, 129, 64, 0] + [9] * 500, 2000, True),
    "16_lanes": ([65, 66, 250, 256] * 400 + [3] * 300, 60000, True),
    "8_lanes": ([65, 71, 72, 73, 256, 2] * 600, 90000, True),
    "8_lanes_no_team": ([65, 130, 256, 257, 300, 2] * 600 + [1500, 1024, 1025], 90000, False),
    "only_wide": ([100] * 37, 500, True),
    # a front in which rows of up to 2,048 are not cut
    "whole_rows": ([2048] * 700 + [2049] * 600 + [1025, 1500, 3000] * 40, 20000, False),
}


@pytest.mark.parametrize("shape", SHAPES)
def test_fixed_iterations_match_oracle(oracle, shape):
    lengths, n, team = SHAPES[shape]
    prob = _lp(lengths, n, 19)
    p = params(oracle, eps=1e-14, iteration_limit=250)
    got = cp.solve(prob, p)
    ref, _ = ol.oracle_solve(oracle, prob, p)
    assert (got.info["graphs"] == 0) == team
    assert got.result["total_count"] == ref["total_count"]
    for key in ("x", "y"):
        a, b = got.result[key], np.asarray(ref[key])
        # FP64 rounding alone: 250 non-expansive iterations of sums of up to 1,500 terms
        assert np.max(np.abs(a - b)) <= 1e-9 * (1.0 + np.max(np.abs(b))), key


@pytest.mark.parametrize("shape", SHAPES)
def test_infinity_norm_matches_oracle(oracle, shape):
    lengths, n, _ = SHAPES[shape]
    prob = _lp(lengths, n, 23)
    p = params(oracle, eps=1e-14, iteration_limit=250)
    p.optimality_norm = cp.NORM_LINF
    got = cp.solve(prob, p).result
    ref, _ = ol.oracle_solve(oracle, prob, p)
    for key in ("relative_primal_residual", "relative_dual_residual"):
        assert abs(got[key] - ref[key]) <= 1e-8 * (1e-3 + abs(ref[key])), key


@pytest.mark.parametrize("shape", ["32_lanes", "8_lanes_no_team", "long_columns"])
def test_rescaling_is_exact(lib, oracle, shape):
    if shape == "long_columns":  # A^T's rows: 40 of a few hundred to a few thousand
        lengths, n = [12] * 5000, 40
    else:
        lengths, n, _ = SHAPES[shape]
    prob = _lp(lengths, n, 29)
    p = ol.oracle_params(oracle)
    g, o = _gpu_rescale(lib, prob, p), ol.oracle_rescale(oracle, prob, p)
    # maxima, square roots, divisions and sums in the rows' order: the same bits
    for k in ("vals", "con", "var"):
        assert np.array_equal(g[k], o[k]), k
