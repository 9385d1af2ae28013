"""The scratch buffers that plans share (tests/cpu_solver/scratch_pool.cu, on the CPU): calls one after another share
one; plans at work together have one each and go back to it without waiting for the others; a plan that finds none
free, or that has lost its own, waits for the work in the one that it gets; so does a plan at the address of one that
has gone."""
import json

import pytest

from test_solver_core import _build_and_run


def test_who_gets_which_buffer(tmp_path_factory):
    d = json.loads(_build_and_run(tmp_path_factory, "scratch_pool", ("-gencode", "arch=compute_103a,code=sm_103a")))
    if d["gpu"]:
        pytest.skip("events that are stand-ins: for machines without a GPU")
    assert d["most"] == 4
    assert len(set(d["one_by_one"])) == 1 and d["held"] == 1
    assert len(set(d["together"])) == d["most"]
    assert d["again"] == d["together"] and d["again_waits"] == 0
    assert d["over"] in d["together"] and d["over_waits"] == 1
    assert d["displaced_waits"] == 1
    assert d["next_waits"] == 1
    assert d["live"] == 0
