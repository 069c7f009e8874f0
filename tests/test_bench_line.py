"""bench.py's line on stdout: every key of the benchmark's contract, numbers as
they were measured, and short; and the byte counts of the kernels a step launches."""
import json
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))


def _full():
    value = {"value": 12345678.123456789, "unit": "cell-updates/s", "trials": [1.0] * 3, "timing": "x" * 80}
    e2e = {**value, "h2d_bytes_per_step": 14680064, "d2h_bytes_per_step": 12582912}
    roof = {k: 1234.123456789012 for k in ("bound", "achieved", "peak", "unit", "frac", "traffic", "kernel", "kernel_ms",
                                           "share_of_step", "limiter")}
    full = {k: 112618048.25471014 for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                                            "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "gpu_launches")}
    full.update(config={k: "y" * 110 for k in ("workload", "precision", "method", "parallelism", "l2", "bytes_note",
                                               "bytes_per_cell_update")},
                clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 1}, e2e=e2e, roofline=roof,
                cpu_baseline={**value, "cores": 16, "kind": "port", "sample": "z" * 200}, node_kernel={"ms": 1.0})
    for k in ("module_step", "pageable", "module_step_pageable", "device_forcing"):
        full["e2e_" + k] = e2e
    full["variants"] = {k: {**value, "fp64": value, "fp32": value, "plain_fp32": value, "note": "w" * 500}
                        for k in ("plain_fp64", "plain_fp64_pairs", "distorted_mixed", "ensemble32", "learned_fp32", "bbm",
                                  "spherical", "ice_growth")}
    full["velocity_error_vs_fp64"] = {k: {"u_v_rms_m_per_s": 0.0037} for k in ("fp32", "fp64_h_times_1p1e-14")}
    return full


def test_every_key_and_short():
    import bench
    full = _full()
    line = bench.headline(full)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline"):
        assert key in line, key
    assert line["value"] == full["value"] and line["e2e"]["value"] == full["e2e"]["value"]
    assert line["e2e"]["h2d_bytes_per_step"] == 14680064 and line["e2e"]["d2h_bytes_per_step"] == 12582912
    assert line["e2e_other"]["module_step"] == full["e2e_module_step"]["value"]
    assert line["variants"]["plain_fp64"] == full["variants"]["plain_fp64"]["value"]
    assert len(json.dumps(line)) < 3000


@pytest.mark.parametrize("kind,word,spherical,expected", [
    ("fp64", 8, False, 16 + 72 + 288 + 64),           # tensor grid: rho and 1 / k_x^2
    ("affine", 4, False, 16 + 72 + 144 + 32),         # four coefficients
    ("global", 4, False, 180 + 72 + 144 + 32),        # 36 derivatives and 9 of the projection
    ("global", 4, True, 216 + 72 + 144 + 32),         # and 9 metric terms
    ("global", 8, True, 432 + 12 + 72 + 288 + 64),    # and three exponents
    ("tma", 4, False, 1580), ("pairs", 8, False, 3016)])
def test_launched_stress_bytes(kind, word, spherical, expected):
    import bench
    assert bench.launched_stress_bytes(kind, word, spherical) == expected


def test_fp64_node_streams():
    """Eight FP64 values read, two written and a flag per node."""
    import bench
    from nextsimdg_gb300.boxtest import BoxTest
    box = BoxTest(16)
    node = bench.launched_bytes_per_cell_update(box, 0, "fp64")["per_iteration_node_share"]
    assert node == pytest.approx(33 * 33 * 81 / 256)
