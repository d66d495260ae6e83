"""CPU-only: the table of DRAM counters that the benchmark reads beside its measurements."""
import json
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_dram_traffic_table():
    """One record per width of the sweep, of plausible size, and none for another graph.  A table taken with other kernel code is
    dropped by the benchmark, whose line then has no bandwidth: that is the skip below, until it is captured again (the
    command is in the table)."""
    import bench
    rec = json.load(open(os.path.join(ROOT, "profiles", "dram_traffic.json")))["aggregation"]["spmm_sweep"]
    assert bench.measured_traffic(rec["nnz"] + 1, bench.WIDTHS) is None
    for f in bench.WIDTHS:       # at least x and y once, at most the indices and every gathered row
        assert 8 * 2**rec["scale"] * f <= rec["bytes"][str(f)] <= rec["nnz"] * (8 + 4 * f)
    if rec["code_sha256"] != bench.aggregation_code_sha256():
        pytest.skip("profiles/dram_traffic.json is of other kernel code: capture it again")
    assert bench.measured_traffic(rec["nnz"], bench.WIDTHS) == {f: rec["bytes"][str(f)] for f in bench.WIDTHS}
