"""The bench's FP64 entry names what bounds the FP64 passes and gives no
fraction of a peak that does not."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fp64_roofline_entry():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    r = bench.fp64_roofline(500, 3500.0)
    assert r["bound"] == "int_mad" and r["achieved"] == 500 * 3500.0 * 1e6 / 1e12
    assert "frac" not in r and "peak" not in r
