"""The step kernels of a large matrix whose rows have at most two entries (the
columns of an LP here, from none to two entries each): points against the CPU
oracle.  (Their FP32 sums: test_gpu_fp32_sums.py.)"""
import numpy as np
import pytest

import cupdlpx as cp
import oracle_lib as ol
from test_gpu_solve import params

pytestmark = pytest.mark.gpu


def _narrow(n, m, seed):
    rng = np.random.default_rng(seed)
    count = np.minimum(2, rng.integers(0, 20, n))  # mostly 2, some 0 and 1
    col = np.repeat(np.arange(n), count)
    row = rng.integers(0, m, len(col))
    order = np.lexsort((col, row))
    row, col = row[order], col[order]
    ptr = np.zeros(m + 1, dtype=np.int64)
    ptr[1:] = np.bincount(row, minlength=m).cumsum()
    val = rng.choice([1.0, -1.0, 0.5], len(col))
    act = np.bincount(row, weights=val * rng.random(n)[col], minlength=m)
    return cp.Problem.from_csr(ptr, col, val, n, c=rng.uniform(-1, 1, n), lc=act - rng.random(m),
                               uc=np.where(rng.random(m) < 0.3, act, np.inf), lv=np.zeros(n),
                               uv=np.where(rng.random(n) < 0.8, 10.0, np.inf))


def test_narrow_steps_match_oracle(oracle):
    prob = _narrow(2500001, 90001, 3)
    p = params(oracle, eps=1e-14, iteration_limit=90)
    p.sv_max_iter = 20
    got = cp.solve(prob, p).result
    ref, _ = ol.oracle_solve(oracle, prob, p)
    assert got["total_count"] == ref["total_count"]
    for key in ("x", "y"):
        a, b = got[key], np.asarray(ref[key])
        # FP64 rounding over 90 iterations
        assert np.max(np.abs(a - b)) <= 1e-9 * (1.0 + np.max(np.abs(b))), key
