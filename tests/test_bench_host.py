"""bench.py's entries that need no GPU."""
import importlib


def test_batch_roofline_names_no_fraction_of_a_peak_it_does_not_use():
    bench = importlib.import_module("bench")
    loop = bench.batch_roofline(True, 8946.0, 6484.0)
    assert loop["bound"] == "latency" and loop["peak"] is None and loop["frac"] is None
    step = bench.batch_roofline(False, 3242.0, 6484.0)
    assert step["bound"] == "hbm" and step["frac"] == 0.5
