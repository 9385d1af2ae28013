"""The translations without atomics after an allocation that failed (tests/cpu_solver/owner_retry.cu, on the CPU):
the call says so, the next one succeeds, and nothing is left behind when the plan goes."""
import json

import pytest

from test_solver_core import _build_and_run


def test_failed_allocations_leave_nothing(tmp_path_factory):
    d = json.loads(_build_and_run(tmp_path_factory, "owner_retry", ("-gencode", "arch=compute_103a,code=sm_103a")))
    if d["gpu"]:
        pytest.skip("kernels on host memory: for machines without a GPU")
    assert {r["type"] for r in d["runs"] if r["failed"]} == {0, 1, 2}
    for r in d["runs"]:
        assert (r["status"] != 0) == bool(r["failed"]), r
        assert r["again"] == 0 and r["left"] == 0, r
