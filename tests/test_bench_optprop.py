"""The benchmark's optical-property section without a reference (CPU only)."""
import argparse
import sys

from conftest import REPO

sys.path.insert(0, REPO)


def test_times_stay_without_a_reference(monkeypatch):
    """A reference run that fails costs its own columns, not the section."""
    import bench
    from jscat import api
    from oracle import refrun

    def fails(*a, **kw):
        raise RuntimeError("reference run failed")

    monkeypatch.setattr(api, "read_aero", lambda ctl, f, d=None: None)
    monkeypatch.setattr(api, "get_opt_prop", lambda ctl, aero: None)
    monkeypatch.setattr(refrun, "reference_aero", fails)
    out = bench.optprop_bench(argparse.Namespace(jacobians=3), None, cpu=True)
    assert len(out["cases"]) == 3
    for row in out["cases"]:
        assert row["ms"] >= 0 and row["reference_error"] == "reference run failed"
        assert "reference_cpu_ms" not in row
