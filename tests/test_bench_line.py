"""bench.py's result line: one JSON object that a log's tail of 1500 characters holds
whole, with the run's figures to 7 digits, however much else was measured."""
import importlib.util
import json
import pathlib

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_mod", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def _full(bench, world):
    x = 7021388191.104858
    kernels = {k: 1.0184213717778523 / 3 for k in ("bin_count", "bin_scan", "bin_scatter", "bin_fixup", "g2p", "p2g")}
    return {
        "metric": bench.METRIC, "value": x * world, "unit": "particle-steps/s", "n_gpus": world, "steps": 20,
        "warmup": 5, "ms_per_step": 2.3894123458862305, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded cube3d scene, numpy PCG64)",
        "config": {"workload": "cube3d: unit cube 256^3 cells, centre cube side 0.5 at 2^3 particles/cell, "
                               "Neo-Hookean E=1e6 nu=0.3, gravity, dt=5e-5; one MPM step per bench step",
                   "n_particles": 16777216, "scale": 1, "form": "f" * 90,
                   "parallelism": "1 GPU" if world == 1 else f"replicas x{world}",
                   "l2": "inputs larger than L2 (3.1 GB particle state per replica)", "particle_order": "o" * 250},
        "accuracy": {"steps": 100, "rel_err_x": 1.2345678901234e-8, "rel_err_v": 9.87654321e-7,
                     "fullsize_oracle_check": {"note": "n" * 300}},
        "configs": {c: {"forms": {f: kernels for f in "abc"}} for c in ("clusters3d", "sphere3d", "dambreak3d")},
        "fp64_plain": {"value": x / 2, "ms_per_step": 5.1},
        "adjoint_over_forward": {"value": 5.123456789, "backward_over_forward": 3.987654321, "fd_check": kernels},
        "roofline": {"bound": "hbm", "kernel": "p2g", "achieved": 1109.9547532353497, "peak": 6552.3, "unit": "GB/s",
                     "frac": 0.16939925724331145, "peak_source": "measured", "traffic": 1288825733.12},
        "kernels_ms_per_step": kernels,
        "cpu_baseline": {"value": 14266903.854666555, "unit": "particle-steps/s", "cores": 16, "kind": "port",
                         "sample": "s" * 170},
        "e2e": {"value": 1462002712.3605003 * world, "unit": "particle-steps/s", "h2d_bytes_per_step": 2281701376,
                "d2h_bytes_per_step": 2885681152, "mpm_steps_per_call": 10, "note": "n" * 90,
                "one_step_per_call": {"value": 177914548.92365032}},
        "gpu_launches": 182,
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 4, "source": "nvml"},
    }


@pytest.mark.parametrize("world", [1, 8])
def test_line_fits_a_log_tail(bench, world):
    out = _full(bench, world)
    if world > 1:
        out["adjoint_over_forward"] = out["cpu_baseline"] = None
    text = bench.result_line(out)
    assert "\n" not in text and len(text) <= 1500
    line = json.loads(text)
    assert set(line) == set(bench.LINE_KEYS)
    for k in ("value", "ms_per_step"):
        assert line[k] == pytest.approx(out[k], rel=1e-6)
    for k in ("metric", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "dtype", "data",
              "gpu_launches", "vs_baseline"):
        assert line[k] == out[k]
    assert line["config"]["workload"] == out["config"]["workload"]
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(line["e2e"])
    assert line["e2e"]["h2d_bytes_per_step"] == out["e2e"]["h2d_bytes_per_step"]
    assert line["clocks"] == {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]}


def test_an_overlong_line_drops_what_is_spare(bench):
    out = _full(bench, 1)
    out["data"] = "d" * 400
    text = bench.result_line(out)
    assert len(text) <= 1500
    assert json.loads(text)["value"] == pytest.approx(out["value"], rel=1e-6)
