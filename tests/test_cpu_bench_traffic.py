"""bench.py reports a kernel's DRAM traffic only from a capture of that kernel."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_traffic_is_of_the_kernel_that_ran(tmp_path, monkeypatch):
    record = {"lp": {"fp32": {"primal_step": {"fused": {"dram_bytes_per_launch": 123}}}}}
    os.makedirs(tmp_path / "profiles")
    (tmp_path / "profiles" / "ncu_traffic.json").write_text(json.dumps(record))
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench.load_traffic("lp", "fp32", "primal_step", "fused") == 123.0
    assert bench.load_traffic("lp", "fp32", "primal_step", "strip") is None
    assert bench.load_traffic("lp", "fp32", "dual_step", "fused") is None
    assert bench.load_traffic("other", "fp32", "primal_step", "fused") is None


def test_every_record_names_its_kernel():
    with open(os.path.join(ROOT, "profiles", "ncu_traffic.json")) as f:
        records = json.load(f)
    for by_precision in records.values():
        for by_step in by_precision.values():
            for by_kernel in by_step.values():
                assert set(by_kernel) <= set(bench.SPMV_KERNELS)
                assert all(r["dram_bytes_per_launch"] > 0 for r in by_kernel.values())
