"""Lists and work units of the batched passes are on the device when their makers return
(tests/cpu_solver/uploads_wait.cu, on the CPU)."""
import json

import pytest

from test_solver_core import _build_and_run


def test_uploads_wait(tmp_path_factory):
    d = json.loads(_build_and_run(tmp_path_factory, "uploads_wait", ("-gencode", "arch=compute_103a,code=sm_103a")))
    if d["gpu"]:
        pytest.skip("kernels on host memory: for machines without a GPU")
    assert d["copies"] >= 6
    assert d["left"] == [[0, 0, 0, 0], [0, 0, 0, 0]]
