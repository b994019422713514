"""The bench's line on stdout: the contract's keys as the full record has them, and
short enough for a reader that keeps the last 3,000 characters, whatever the
figures and however long the record (candidates, checks) is."""
import json

import numpy as np

import bench

W = -1.2345678901234567e-105  # as long as a float prints


def voll():
    form = {"value": W, "ms_per_step": W, "cg_iterations_per_step": W, "pcg_us_per_iteration": W}
    paar = {"mixed_storage": W, "mixed_fp32_vectors": W}
    e2e = {"value": W, "unit": "vertex-steps/s", "h2d_bytes_per_step": 10 ** 9, "d2h_bytes_per_step": 10 ** 9}

    class S:
        n = 10 ** 6
        membran_punkte = biegung_punkte = naht_punkte = np.zeros((10 ** 6, 1))

    return {
        "metric": bench.METRIC, "value": W, "unit": bench.UNIT, "n_gpus": 8, "steps": 1000, "warmup": 100,
        "ms_per_step": W, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
        "data": "synthetic", "config": bench.workload_config(257, S, {"precision": "x" * 88}), "e2e": e2e,
        "gpu_launches": 10 ** 6, "cg_iterations_per_step": W, "pcg_us_per_iteration": W,
        "roofline": {
            "bound": "hbm", "achieved": W, "peak": W, "unit": "GB/s", "frac": W, "kernel": "k" * 35, "note": "n" * 200},
        "clocks": {"sm_mhz": W, "sm_max_mhz": W, "reasons": ["sw_power_cap", "sw_thermal_slowdown"], "samples": 1000},
        "fp64": form, "mixed_fp32_vectors": form,
        "mixed_vs_fp64": {"speedup": paar, "rel_pos_err_after_100_steps": paar, "one_step_error": {
            "errors": {k: [{"max": W, "rms": W}] * 50 for k in paar}}},
        "batched": {"batched_mixed": form, "batched_vs_per_instance": W},
        "launch_shapes": {"candidates": [form] * 100},
        "adjoint": {"forward_ms": W, "backward_ms": W, "backward_forward": W, "gradient_check": {
            "params": [form] * 20, "max_best_rel_err": W}},
        "garment": {"e2e": e2e, **{k: form for k in (
            "selfcollision_mixed_storage", "selfcollision_fp64", "no_selfcollision_mixed_storage",
            "no_selfcollision_fp64")}},
        "mesh": {"nearest": {"ms_device": W, "e2e": {"ms": W}}, "sdf_band_3cm": {"ms_device": W},
                 "step_mesh_body": {"ms_per_step": W}, "step_grid_body": {"ms_per_step": W}},
        "cpu_baseline": {"value": W, "unit": bench.UNIT, "cores": 1, "kind": "port", "sample": "s" * 300}}


def test_laenge_und_schluessel():
    f = voll()
    zeile = bench.line_of(f)
    assert len(json.dumps(zeile)) < 2800
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert zeile[k] == f[k], k


def test_ohne_nebenmessungen():
    f = {k: v for k, v in voll().items() if k not in (
        "fp64", "mixed_fp32_vectors", "mixed_vs_fp64", "batched", "launch_shapes", "adjoint", "garment", "mesh",
        "cpu_baseline")}
    assert bench.line_of(f)["value"] == f["value"]
