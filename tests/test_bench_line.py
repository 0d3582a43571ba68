"""The line bench.py prints stays readable from its last 10,000 characters: with more Poisson variants and steps than a run
has, it is shorter than that, keeps every key and value of the contract, and the rest goes to stderr."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
import bench  # noqa: E402


def full_line():
    variant = {"ms_mean": 12.345678901234567, "cycles_mean": 7.333333333333333, "rel_max": 9.312321986903205e-07,
               "cycles": [7, 7, 8], "ms": [4.007, 4.053, 4.562], "convergence_factor_mean": 0.14196010958687585}
    poisson = {"timed_steps": {"method": "fcg", "ms_mean": 4.63, "cycles_mean": 8.0, "history_last_step": [0.1] * 9},
               "tolerance": 1e-6, "fp32_wcycle": {"reaches_tol": False, "ms_per_cycle": 1.45, "note": "x" * 200},
               **{f"fcg_fp16_c0_s12_w18_cs10_{i}": dict(variant) for i in range(60)},
               "speedup_learned_vs_plain_fcg": 0.67, "learned_at_timed_settings": {"speedup": 0.64, "ms_plain": 8.0}}
    steps = [{"cycles": 8, "rel_residual": 2.650023377315679e-07, "rel_l2_error": 1.4912662584497485e-08,
              "reference_rel_residual": 9.785253676039634e-12}] * 100
    line = {"metric": "steps/s", "value": 140.98546334804982, "unit": "steps/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 7.09, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": {"workload": "w", "note": "x" * 600}, "solver": {"pressure": "x" * 450},
            "parity": {"scene": "x" * 450}, "pressure_error": {"reference": "x" * 250, "steps": steps, "rel_l2_error_max": 2e-8},
            "poisson": poisson, "e2e": {"value": 40.7, "path": "x" * 400}, "roofline": {"kernel": "x" * 400},
            "rooflines": [{"kernel": "x" * 280}] * 6, "cpu_baseline": {"sample": "x" * 250},
            "clocks": {"sm_mhz": 1965.0, "reasons": []}, "gpu_launches": 7180}
    return line


def test_printed_line_is_short_and_complete():
    line = full_line()
    assert len(json.dumps(line)) > 20000
    short, details = bench.printed_line(line)
    assert len(json.dumps(short)) < 10000
    assert short.keys() == line.keys()
    for key in line.keys() - {"poisson", "pressure_error"}:
        assert short[key] == line[key]
    assert len(short["poisson"]["variants_ms"]) == 60 and short["poisson"]["timed_steps"]["ms_mean"] == 4.63
    assert short["pressure_error"] == {"reference": "x" * 250, "rel_l2_error_max": 2e-8}
    assert details == {"poisson": line["poisson"], "pressure_error": line["pressure_error"]}


def test_kernel_names():
    assert bench.update_kernel(2_299_999) == "k_particle_update" and bench.update_kernel(2_300_000) == "k_particle_update_tiled"
    assert [bench.p2g_kernel(True, c) for c in (100_000, 3_499_999, 3_500_000)] == ["k_p2g_gather", "k_p2g_ordered", "k_p2g_tiled"]
