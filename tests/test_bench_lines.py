"""What bench.py says about a field launch: no share of a peak for a sum whose
terms were not all formed, and the FP64 pipe's measured share only from a profile of
the kernels that ran."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

@pytest.fixture
def roof(monkeypatch):
    monkeypatch.setattr(bench, "fp64_peak_tflops", lambda torch: 37.0)
    monkeypatch.setattr(bench, "fp32_peak_tflops", lambda torch: 70.0)
    monkeypatch.setattr(bench, "pipe_peak_tflops", lambda torch, clk, fp64=True: (37.0 if fp64 else 74.0, "test"))

    def make(cells, workload, fp64=True):
        return bench.field_roofline(None, {}, fp64, 1e12, 128, 1.0, cells, workload, traffic=5.0)
    return make


def test_by_cells(roof):
    for workload, low, high in (("fcc_random", 0.6, 0.8), ("bcc_prismatic", 0.6, 0.8)):
        r = roof(True, workload)
        assert r["achieved"] is None and r["frac"] is None and r["frac_of_gemm"] is None and r["traffic"] is None
        assert r["term_by_term_equivalent"] == 128.0
        assert low < r["fp64_pipe_active"] < high and r["fp64_pipe_source"]
    assert roof(True, "fcc_random")["fp64_pipe_source"] != roof(True, "bcc_prismatic")["fp64_pipe_source"]
    assert roof(True, "quadrupole")["fp64_pipe_active"] is None


def test_term_by_term(roof):
    r = roof(False, "fcc_random")
    assert r["achieved"] == 128.0 and r["frac"] == 128.0 / 37.0 and r["traffic"] == 5.0
    assert "form" not in r and "fp64_pipe_active" not in r


def test_no_profiler():
    class NoProfiler:
        class cuda:
            @staticmethod
            def synchronize():
                raise RuntimeError("none here")
    assert bench.kernels_per_call(NoProfiler, lambda: None) is None
