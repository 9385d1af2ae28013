"""The source rows that the dense tensor-core passes copy, against integers of any size: expansions of more than 64 GB
(many columns) lie behind the 2^32nd 16 bytes (tests/cpu_solver/dense_rows.cu, on the CPU)."""
import json

from test_solver_core import _build_and_run


def test_row_copies(tmp_path_factory):
    out = _build_and_run(tmp_path_factory, "dense_rows", ("-gencode", "arch=compute_103a,code=sm_103a"))
    lines = [json.loads(line) for line in out.splitlines()]
    assert len(lines) == 8 * 4 * 3 * 3
    for row, P2, c0, cnt, start, n in lines:
        if row < 0:
            assert n == 0
            continue
        first = row * P2 + c0
        assert start == first // 2
        # the words hold all coefficients and at most one before and one after them
        assert 2 * start + 2 * n >= first + cnt and 2 * n <= cnt + 2
