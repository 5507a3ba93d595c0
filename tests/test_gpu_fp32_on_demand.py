"""The order of a resident problem's FP32 sums is made by its first FP32 solve:
two first solves at once, on a problem uploaded without it, return the bits of a
solve whose upload made it."""
import threading

import numpy as np
import pytest

import cupdlpx as cp
from test_gpu_solve import params
from test_gpu_strip import SHAPES, _lp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["strip_or_front", "item_or_chunks", "two_lanes"])
def test_two_first_solves_at_once(oracle, shape):
    lengths, n = SHAPES[shape]
    prob = _lp(lengths, n, 3)
    p = params(oracle, eps=1e-14, iteration_limit=400)
    ref = cp.solve(prob, p, precision=cp.PRECISION_FP32_REFINE).result
    dp, got = cp.DeviceProblem(prob), [None, None]

    def run(i):
        got[i] = dp.solve(p, precision=cp.PRECISION_FP32_REFINE).result

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    dp.free()
    for r in got:
        assert r["total_count"] == ref["total_count"]
        assert np.array_equal(r["x"], ref["x"]) and np.array_equal(r["y"], ref["y"])
