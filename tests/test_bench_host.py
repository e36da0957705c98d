"""CPU tests of bench.py's host-side pieces: the clock record taken during the timed region and
the roofline denominator."""
from __future__ import annotations

import json

import bench


def _sampler(lines):
    s = bench.ClockSampler(0)
    s.lines = list(lines)
    return s


def test_clock_summary_takes_the_median_and_the_active_reasons():
    lines = [
        "0, 1965, 1965, 700.1, 0x0000000000000000, Not Active, Not Active, Not Active, Not Active",
        "0, 1800, 1965, 990.0, 0x0000000000000004, Not Active, Not Active, Not Active, Active",
        "0, 1950, 1965, 820.5, 0x0000000000000000, Not Active, Not Active, Not Active, Not Active",
        "garbage line",
        "0, [N/A], 1965, 0, 0x0, Not Active, Not Active, Not Active, Not Active",
    ]
    d = _sampler(lines).summary()
    assert d == {"sm_mhz": 1950.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 3}


def test_clock_summary_flags_thermal_and_hardware_slowdowns():
    lines = ["0, 1400, 1965, 1000, 0x68, Active, Active, Active, Not Active"] * 4
    d = _sampler(lines).summary()
    assert d["reasons"] == ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown"]
    assert d["sm_mhz"] == 1400.0


def test_clock_summary_without_samples():
    d = _sampler([]).summary()
    assert d == {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}


def test_roofline_peak_comes_from_the_measured_file(tmp_path, monkeypatch):
    monkeypatch.setattr(bench, "ROOT", tmp_path)
    assert bench._peaks() == (6650.0, "fallback")
    (tmp_path / "MEASURED_PEAKS.json").write_text(json.dumps({"hbm_gbs": 7012.5}))
    assert bench._peaks() == (7012.5, "measured")


def test_headline_is_short_and_keeps_the_contract():
    """The legs' lists stay out of the printed line, which fits the tail of a log; the keys that the
    result is read by are all in it."""
    big = {"walls_s": [0.123456789] * 2000, "ms_per_solve": 1.5, "batch_lps_per_s": 2.5,
           "adjoint_ms_per_instance": 3.5, "nested": {"x": [1] * 1000}}
    line = {"metric": bench.METRIC, "value": 3.4, "unit": bench.UNIT, "n_gpus": 1, "steps": 20,
            "warmup": 5, "ms_per_step": 293.0, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32/f64 mixed", "precision": "p" * 80, "data": "d" * 70,
            "config": {"workload": "w" * 100, "parallelism": "replicas x1"}, "objective_bound": "b" * 200,
            "fp64": big, "mixed_refined_to_1e-8": big, "fp64_to_1e-8": big, "c0": big, "c2": big,
            "batch_c3": big, "batch_c3_mixed": big, "adjoint_c4": big, "iteration_loop": big,
            "roofline": {"bound": "hbm", "achieved": 1.0, "peak": 2.0, "frac": 0.5, "sweeps": big},
            "cpu_baseline": {"value": 0.03, "sample": "s" * 150},
            "e2e": {"value": 3.4, "unit": bench.UNIT, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2,
                    "status": [1] * 20},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []}, "gpu_launches": 9}
    text = json.dumps(bench.headline(line))
    out = json.loads(text)
    assert len(text) < 2500
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
              "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e", "clocks",
              "gpu_launches", "cpu_baseline"):
        assert k in out
    assert out["e2e"]["status"] == [1] and out["batch_c3"] == {"batch_lps_per_s": 2.5}
    assert out["roofline"]["frac"] == 0.5 and "sweeps" not in out["roofline"]
    assert bench.headline({**line, "adjoint_c4": None, "cpu_baseline": None})["value"] == 3.4
