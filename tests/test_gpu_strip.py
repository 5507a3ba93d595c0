"""The strip-format SpMV and the resident team inside whole solves, against
the CPU oracle at a fixed iteration count: matrices whose rows and columns sit
at the edges of the format (64 | 65 non-zeros: strip or front; 1,024 | 1,025:
item or chunks; empty rows and columns; one row), at each number of lanes a
row can have, below and above the size that runs as a team.

FP64 PDHG is the same algorithm on both sides, so the points differ by
rounding alone; over a few hundred non-expansive iterations of FP64 sums of up
to 5,000 terms that stays below 1e-9 of the largest entry."""
import numpy as np
import pytest

import cupdlpx as cp
import oracle_lib as ol
from test_gpu_solve import params

pytestmark = pytest.mark.gpu


def _lp(lengths, n, seed):
    """Rows of the given lengths over n columns, a feasible point, mixed bounds."""
    rng = np.random.default_rng(seed)
    m = len(lengths)
    ptr = np.zeros(m + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(lengths)
    if max(lengths) > n // 4:
        col = np.concatenate([np.sort(rng.choice(n, L, replace=False)) for L in lengths])
    else:  # random columns, duplicates allowed
        col = rng.integers(0, n, ptr[-1])
    val = rng.standard_normal(ptr[-1])
    x0 = rng.random(n)
    act = np.add.reduceat(np.append(val * x0[col], 0.0), np.minimum(ptr[:-1], ptr[-1]))
    act = np.where(np.diff(ptr) > 0, act, 0.0)
    eq = rng.random(m) < 0.3
    return cp.Problem.from_csr(ptr, col, val, n, c=rng.uniform(-1, 1, n),
                               lc=np.where(eq, act, act - rng.random(m)),
                               uc=np.where(eq, act, np.inf), lv=np.zeros(n),
                               uv=np.where(rng.random(n) < 0.8, 10.0, np.inf))


def _edges(*special, rest=0, count=0):
    return list(special) + [rest] * count


SHAPES = {
    "one_row": (_edges(7), 9),
    "strip_or_front": (_edges(64, 65, 63, 0, 1, 64, rest=3, count=40), 200),
    "item_or_chunks": (_edges(1024, 1025, 2048, 2049, 66, 5000, 0, rest=5, count=300), 6000),
    "packed_front": (_edges(rest=70, count=37), 500),
    "eight_lanes": (_edges(0, 33, rest=9, count=4000), 5003),
    "two_lanes": (_edges(0, 33, rest=7, count=15001), 17000),
    "one_lane": (_edges(0, 33, rest=6, count=45001), 50021),
    "no_team": (_edges(0, 70, 1500, rest=14, count=301003), 400007),
}


@pytest.mark.parametrize("shape", SHAPES)
def test_fixed_iterations_match_oracle(oracle, shape):
    lengths, n = SHAPES[shape]
    prob = _lp(lengths, n, 17)
    p = params(oracle, eps=1e-14, iteration_limit=250)
    got = cp.solve(prob, p)
    ref, _ = ol.oracle_solve(oracle, prob, p)
    assert got.info["spmv_kernel_A"] == got.info["spmv_kernel_AT"] == 2
    assert got.result["total_count"] == ref["total_count"]
    for key in ("x", "y"):
        a, b = got.result[key], np.asarray(ref[key])
        assert np.max(np.abs(a - b)) <= 1e-9 * (1.0 + np.max(np.abs(b))), key


def test_infinity_norm_matches_oracle(oracle):
    prob = _lp(SHAPES["item_or_chunks"][0], 6000, 23)
    p = params(oracle, eps=1e-14, iteration_limit=250)
    p.optimality_norm = cp.NORM_LINF
    got = cp.solve(prob, p).result
    ref, _ = ol.oracle_solve(oracle, prob, p)
    for key in ("relative_primal_residual", "relative_dual_residual"):
        assert abs(got[key] - ref[key]) <= 1e-8 * (1e-3 + abs(ref[key])), key
