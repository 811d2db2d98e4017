"""bench.py's rate of the group pass: the counted operations are those of the
reference's algorithm, so they give no share of a peak."""
import bench


def test_group_pass_rate_claims_no_share_of_the_peak(monkeypatch):
    monkeypatch.setattr(bench, "fp64_peak_tflops", lambda: {"tflops": 30.0, "source": "test"})
    r = bench.group_pass_rate(2e9, 1.0)
    assert r["kernel"] == "k_cp<12>" and r["frac"] is None
    assert abs(r["achieved"] - 2.0) < 1e-12
