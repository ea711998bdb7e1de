"""The benchmark's JSON line stays short enough for a reader that keeps the last few KB of the output,
with every key of the contract, whatever the legs' per-step lists hold."""
import json
import sys
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent

CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "e2e", "roofline", "cpu_baseline")


def _arm(steps):
    return {"value": 123.456789012345, "ms_per_step": 8.1234567890123, "steps": steps,
            "iterations_per_step": 376.123456789, "speedup_vs_fp64": 1.723456789012,
            "rel_err_vs_fp64_1e-13_max": {"face_traces": 8.426916744853071e-09, "cell_values": 8.4e-09},
            "rel_err_vs_fp64_1e-13_per_step": [8.426916744853071e-09] * steps}


def test_line_is_short_and_whole():
    sys.path.insert(0, str(REPO))
    import bench

    kernel = {"kernel": "k_spmv_dot<double,6,1> (v = A p, (rh, v))", "ms": 0.05178559944033623, "gbs": 5877.1007247033995,
              "hbm_frac": 0.8653739618787584, "bytes": 304349184.0, "share_of_iteration": 0.317723638}
    long = "x" * 180
    protocol = {k: {"protocol": _arm(800), "training_phase": _arm(200), "used_phase": _arm(600),
                    "speedup_vs_fp64": {"protocol": 1.5, "used_phase": 1.9}}
                for k in ("fp64", "mixed", "learned", "learned_mixed", "extrapolation_only", "learned_linear_base",
                          "extrapolation_only_linear")}
    protocol["workload"] = long
    line = {k: 1.23456789012345 for k in CONTRACT}
    line.update({
        "metric": "m" * 90, "unit": "time steps/s", "data": "d" * 100, "dtype": "f64", "n_gpus": 1, "steps": 20, "warmup": 5,
        "config": {"workload": "diffusion3d_64", "cells": 1572864, "faces": 3170304, "rows": 3170304, "l2": "l" * 100},
        "e2e": {"value": 15.363262246412617, "unit": "time steps/s", "h2d_bytes_per_step": 12582912,
                "d2h_bytes_per_step": 12582912, "path": "p" * 70, "steps": "s" * 80},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 7},
        "cpu_baseline": {"value": 0.5059321966669338, "unit": "time steps/s", "cores": 16, "kind": "port", "sample": long},
        "roofline": dict(kernel, traffic_source="t" * 90, selection=long, other_spmv=kernel),
        "iteration_kernels": {k: kernel for k in ("spmv_dot", "update_s", "spmv_dots2", "update_xr", "update_p")},
        "kernels": {k: kernel for k in ("cell_local", "assemble", "reconstruct", "spmv_fp64")},
        "forms": {"mixed": _arm(1000), "fp64_gmres": dict(_arm(3), solver=long), "learned_protocol": protocol},
        "other_cells": {"cuboids": dict(_arm(20), kernels={"assemble": kernel})},
        "other_configs": {"heat2d": {"workload": "heat2d_128", "fp64": _arm(100)},
                          "adr2d": {"workload": "adr2d_512", "fp64": _arm(200)},
                          "mixed128": {"fp64": _arm(20), "mixed": _arm(20), "iterations_per_step_fp64": [1000] * 20}},
    })
    text = json.dumps(bench.result_line(line))
    assert len(text) < 4096
    d = json.loads(text)
    for k in CONTRACT:
        assert k in d
    for k in ("metric", "value", "e2e", "clocks"):
        assert d[k] == bench.rounded(line[k])
    assert d["forms"]["mixed"]["value"] == 123.457 and d["forms"]["learned_protocol"]["learned"] == 123.457
    for legs in (None, {}):  # legs switched off
        bench.result_line(dict(line, forms={}, other_cells=legs, other_configs={}))
