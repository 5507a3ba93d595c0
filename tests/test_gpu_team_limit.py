"""LPs with as many rows as a resident team's warps take two strips of, and with
one more: the second runs a kernel per product (every CTA of a team folds every
strip's partial sums itself).  Both give the oracle's points."""
import numpy as np
import pytest

import cupdlpx as cp
import oracle_lib as ol
from test_gpu_solve import params
from test_gpu_strip import _lp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("more", [0, 1])
def test_team_up_to_two_strips_a_warp(oracle, more):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 2 * sms * 2 * 8 * 32 + more  # two strips a warp, two CTAs of 8 warps an SM
    prob = _lp([2] * rows, rows // 3, 5)
    p = params(oracle, eps=1e-14, iteration_limit=130)
    got = cp.solve(prob, p)
    ref, _ = ol.oracle_solve(oracle, prob, p)
    assert (got.info["graphs"] > 0) == bool(more)
    for key in ("x", "y"):
        a, b = got.result[key], np.asarray(ref[key])
        # FP64 rounding over 130 non-expansive iterations of sums of a few terms
        assert np.max(np.abs(a - b)) <= 1e-9 * (1.0 + np.max(np.abs(b))), key
