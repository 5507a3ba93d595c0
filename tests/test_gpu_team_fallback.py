"""A resident team whose barrier waits run out: the solve takes the launch's work
back, goes on with a kernel per product, and returns the same bits.  The arrival
counter starts where no barrier completes, so that every CTA gives up at its
first one after the wait's limit (2 s)."""
import numpy as np
import pytest

import cupdlpx as cp
from test_gpu_solve import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cp.PRECISION_FP64, cp.PRECISION_FP32_REFINE,
                                       cp.PRECISION_FP32_MATRIX])
def test_solve_goes_on_without_the_team(oracle, monkeypatch, precision):
    prob = cp.Problem.generated("random", 2000, 5000, 20000, 7)
    p = params(oracle, eps=1e-12, iteration_limit=1700)
    team = cp.solve(prob, p, precision=precision)
    monkeypatch.setenv("PDLP_TEAM_FAIL", "1")
    alone = cp.solve(prob, p, precision=precision)
    # the second one really ran as single launches
    assert alone.info["kernel_launches"] > 2000 > team.info["kernel_launches"]
    assert alone.info["power_iterations"] == team.info["power_iterations"]
    assert alone.info["sigma_max"] == team.info["sigma_max"]
    for key in ("status", "total_count", "primal_objective_value", "dual_objective_value",
                "relative_primal_residual", "relative_dual_residual"):
        assert alone.result[key] == team.result[key], key
    for key in ("x", "y", "rc"):
        assert np.array_equal(alone.result[key], team.result[key]), key
