"""The bench reports DRAM traffic only from a capture of the kernel it timed."""
import importlib.util
import os

import helpers as h


def test_no_traffic_without_a_capture():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(h.ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    assert not hasattr(bench, "MEASURED_TRAFFIC_PER_PRIME")  # was another kernel's
    assert bench.hbm_record(None, 1000.0) is None
    rec = bench.hbm_record(2e12, 1000.0)
    assert rec["achieved"] == 2000.0 and rec["frac"] == 2000.0 / rec["peak"]
