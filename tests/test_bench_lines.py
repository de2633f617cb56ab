"""The bench's roofline entry: a fraction of HBM only for kernels that stream the state through it."""
import bench


def test_roofline_entry_of_both_forms(monkeypatch):
    monkeypatch.setattr(bench, "measured_peaks", lambda: (5000.0, "measured"))
    line = bench.roofline_line(1.0, 2_500_000_000, 0, "iterate kernel", 7.0)
    assert line["bound"] == "hbm" and line["frac"] == 0.5 and line["achieved"] == 2500.0
    assert line["traffic"] == 7.0 and line["launch_ms"] == 1.0 and line["algorithmic_bytes_per_launch"] == 2_500_000_000
    line = bench.roofline_line(1.0, 2_500_000_000, 3, "iterate kernel", 7.0)
    assert line["bound"] != "hbm" and line["pairs_on_chip"] == 3 and line["launch_ms"] == 1.0
    assert line["frac"] is None and line["achieved"] is None and line["traffic"] is None
