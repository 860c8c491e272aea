"""The line that bench.py prints: short enough for a log that keeps a few
thousand characters, strict JSON, nothing of the required keys lost (no GPU)."""
import json

import bench

REQUIRED = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "roofline", "e2e")


def _full_line():
    """A line with every leg, each as large as the legs make it."""
    x = 1.2345678901234567
    table = [{"variant": i, "voxels_per_thread": 4, "min_ctas": 4, "regs": 64, "ctas_per_sm": 3, "ms_per_step": x,
              "ms_per_step_min": x, "ms_per_step_max": x} for i in range(27)]
    react = [{"index": i, "voxels": 91292, "max_dlat_steps": 30, "p99_dlat_steps": x} for i in range(8)]
    case = {"first": {"max_dlat_steps": 1, "p99_dlat_steps": x, "voxels_one_run_only": 0}, "reactivations": react,
            "max_abs_dvm_1khz": x, "electrogram": {"rel": x}}
    sample = {"instance": 1, "model": "ms", "first_max_dlat_steps": 1, "max_abs_dvm_1khz": x}
    serving = {"requests": 300, "p50_latency_s": x, "p99_latency_s": x, "throughput_voxel_steps_s": x * 1e10,
               "builder": "b" * 300, "plain_fp64_serial_subset": {"requests": [{"rid": i} for i in range(9)]}}
    return {
        "metric": bench.METRIC, "value": 1.93e10 * x, "unit": "voxel-steps/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded shells; no patient meshes)",
        "config": {"workload": bench.WORKLOAD, "instances": 64, "voxels": 10900000, "steps_per_launch": 10,
                   "pre_steps": 1000, "gmres": "early exit, tol 1e-07, restart 20",
                   "l2": "inputs larger than L2 (no flush)", "parallelism": "instance-parallel x1"},
        "gpu_launches": 2, "autotune": {"variant": 7, "ctas_per_sm": 4, "table": table},
        "solver": {"arnoldi_per_solve": x, "solves_per_step": x, "arnoldi_per_step": x},
        "roofline": {"bound": "hbm", "achieved": 2630.123456789 * x, "peak": 6547.8, "unit": "GB/s", "frac": 0.4 * x,
                     "peak_source": "of measured", "traffic": 1.578e10 * x, "traffic_source": "s" * 150,
                     "kernel": "step_kernel<float,2,4,false,0,true>", "bytes_per_voxel_step": 136.0 * x},
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]},
        "phases_ms_per_step": {"cta_utilization": 0.92, "barriers_per_step": x, "per_instance": [[x] * 7] * 12},
        "e2e": {"value": 1.4e10 * x, "unit": "voxel-steps/s", "h2d_bytes_per_step": 1e5 * x, "d2h_bytes_per_step": 1e7 * x,
                "seconds": 12.7, "run_only_value": 2e10 * x, "path": "p" * 400},
        "e2e_dropin_c1": {"voxels": 40000, "plain_fp64": {"simulate_s": x}, "fast_fp32": {"simulate_s": x}},
        "plain_fp64": {"value": 6e8 * x, "ms_per_step": x, "voxels": 157000, "speedup_batched_fp32": 31.5 * x,
                       "phases_ms_per_step": {str(i): x for i in range(12)}},
        "accuracy": {"reference": "r", "c1": case, "c2_wall3": case, "c2_wall8": case, "c3_sample": [sample] * 4},
        "anisotropic": {"value": 1e10 * x, "ms_per_step": x, "voxels": 2400000, "fibres": "f" * 60},
        "geometry": {"host_numpy_s": x, "device_s": x, "device_s_all": [x] * 3}, "serving": dict(serving),
        "serving_half_load": dict(serving, p99_latency_s=float("nan")),
        "electrogram": {"bf16x3_ms": x, "executed_tflops": 1454.3 * x, "fp64_contract_ms": 93.1 * x, "leadfield_ms": x,
                        "rel_l2_bf16x3_vs_fp64": 1e-4 * x, "tile_config_ms": {str(i): x for i in range(4)}},
        "cpu_baseline": {"value": 2e6 * x, "unit": "voxel-steps/s", "cores": 16, "kind": "port",
                         "sample": "192 steps of instance 42 (175353 voxels, MS) from t=0 in 15.0 s"}}


def test_line_is_short_strict_and_complete():
    full = _full_line()
    assert len(json.dumps(full)) > 6000
    text = json.dumps(bench.short_line(full), allow_nan=False)
    assert len(text) < 3000 and "\n" not in text
    got = json.loads(text)
    assert set(REQUIRED) <= set(got) and set(got) == set(full)
    for k in ("metric", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "dtype", "data",
              "config", "gpu_launches", "clocks"):
        assert got[k] == full[k]
    assert abs(got["value"] / full["value"] - 1) < 1e-6 and abs(got["e2e"]["value"] / full["e2e"]["value"] - 1) < 1e-6
    assert got["serving_half_load"]["p99_latency_s"] is None
    assert got["e2e_dropin_c1"] == {"plain_fp64.simulate_s": 1.234568, "fast_fp32.simulate_s": 1.234568}
    assert got["accuracy"]["c1"]["first_max_dlat_steps"] == 1 and got["accuracy"]["c3_first_max_dlat_steps"] == 1


def test_line_without_extras():
    full = {k: v for k, v in _full_line().items() if k in REQUIRED and k != "e2e"}
    full["autotune"] = None
    assert bench.short_line(full)["autotune"] is None
