"""The line of the whole-run bench is short enough for a reader that keeps the end
of the output, and keeps the keys such a reader needs."""
import json

import bench

CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline")


def whole_run():
    x = 123456.789012345678
    choice = {"neighbour": "cell", "tile_split": 4, "skin": 0.0, "sparse_below": 24.0, "cell_units": 0, "subcells": 0,
              "ms_per_step": x}
    forms = {}
    for name in ("fp32x", "fp32c", "fp64"):
        forms[name] = {"value": x * 1e4, "e2e": x * 1e4, "ms_per_step": x, "ms_per_bench_step": [x] * 20,
                       "profile_ms_final_state": {k: x for k in "abcdef"}, "autotune": [choice] * 12,
                       "retunes": [{"after_step": 500 * k, "choice": choice} for k in range(20)],
                       "order_params_series": [[500 * k, x, x] for k in range(20)]}
        if name != "fp64":
            forms[name]["drift_vs_fp64"] = {"max_dR": 1.2345678901e-12, "max_dR_local": 1.2345678901e-12,
                                            "points": 20, "every_steps": 500}
    phases = {k: 0.0414635798761785 for k in ("stage", "sort", "gather", "pass1", "pass2")}
    config = {"workload": "vortex_srk_n65536_L8", "N": 65536, "L": 8.0, "stepper": "srk",
              "model": "vortex (alignment + natural frequencies)",
              "neighbour": "autotuned per precision (cell list or Verlet rows)", "dt": 0.005,
              "sim_steps_per_bench_step": 500, "l2": "flushed between bench steps (512 MB write, outside the timed events)",
              "parallelism": "replicas1", "run": "x" * 120, "start_state": "x" * 120}
    return {"metric": "particle-steps/s", "value": x * 1e4, "unit": "particle-steps/s", "n_gpus": 1, "steps": 20,
            "warmup": 5, "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32x (f32 pair tests; exact i64 fixed-point neighbour sums; f64 per-particle rates, noise, "
                     "positions, phase)", "data": "synthetic (seeded uniform positions/phases, normal frequencies)",
            "config": config, "form": "fp32c", "drift": forms["fp32c"]["drift_vs_fp64"], "forms": forms,
            "fp32x_over_fp64": x, "fp32c_over_fp64": x, "value_warm_window": x * 1e4, "gpu_launches": 110000,
            "roofline": {"bound": "hbm", "kernel": "pass2", "kernels": ["k" * 40] * 3, "achieved": x, "peak": 6786.2,
                         "peak_kind": "measured", "unit": "GB/s", "frac": 0.02258535655123022, "traffic": 9760000.0,
                         "traffic_state": "x" * 80, "alg_bytes_per_particle": 100, "alg_bytes_per_launch": 6553600,
                         "phase_ms_run_mean": phases, "timing": "x" * 150,
                         "compute": {"candidate_tests_per_s": x * 1e8, "pair_terms_per_s": x * 1e8,
                                     "candidates_per_particle_run_mean": x, "pairs_per_particle_run_mean": x},
                         "note": "x" * 200},
            "e2e": {"value": x * 1e4, "unit": "particle-steps/s", "h2d_bytes_per_step": 1572864,
                    "d2h_bytes_per_step": 1572864,
                    "per_call": "pinned state upload, the bench step's steps, state download"},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"], "samples": 863},
            "cpu_baseline": {"value": x, "unit": "particle-steps/s", "cores": 1, "kind": "port",
                             "sample": "N=65536, 3 SRK steps after one warm step"}}


def test_line_is_short_and_complete():
    out = whole_run()
    line = bench.line_of(out)
    assert len(line) <= bench.LINE_BYTES and "\n" not in line
    got = json.loads(line)
    assert all(k in got for k in CONTRACT)
    assert got["value"] == bench.rounded(out["value"]) and abs(got["value"] / out["value"] - 1) < 1e-6
    assert set(got["forms"]) == {"fp32x", "fp32c", "fp64"} and got["forms"]["fp64"]["value"] > 0
