"""The power method's iteration limit (sv_max_iter) on an LP that a resident team
runs: it ends after exactly that many iterations when the tolerance is out of
reach, and a limit of zero or below runs none and leaves the estimate at zero,
as on an LP that runs a kernel per product."""
import ctypes as C

import numpy as np
import pytest

import cupdlpx as cp
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [-3, 0, 1, 2, 7, 16, 33])
def test_power_method_ends_at_its_limit(lib, oracle, limit):
    prob = cp.Problem.generated("random", 800, 2000, 12000, 5)
    p = ol.oracle_params(oracle)
    p.sv_max_iter, p.sv_tol = limit, 0.0
    s, it = C.c_double(), C.c_int()
    assert lib.pdlp_gpu_power_method(prob.ptr, C.byref(p), C.byref(s), C.byref(it)) == 0
    if limit <= 0:
        assert (it.value, s.value) == (0, 0.0)
        return
    o = ol.oracle_rescale(oracle, prob, p)
    a = prob.arrays()
    v0 = np.zeros(a["m"])
    oracle.oracle_power_start_vector(a["m"], cp.as_dp(v0))
    oit = C.c_int()
    so = oracle.oracle_power_method(a["m"], a["n"], cp.as_ip(a["row_ptr"]), cp.as_ip(a["col_ind"]),
                                    cp.as_dp(o["vals"]), cp.as_dp(v0), limit, 0.0,
                                    C.byref(oit), 0)
    assert it.value == oit.value == limit
    # the same iteration in FP64 on both sides; only the order of the sums differs
    assert abs(s.value - so) <= 1e-12 * so
