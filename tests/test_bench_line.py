"""The bench's launch counts per iteration, against the launch sequences in the
sources, and the length of the line it prints (CPU)."""
import importlib.util
import json
from pathlib import Path

import pytest

from unsflow2d_gb300 import abi

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_line_under_test", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_launches_per_iteration(bench):
    p = abi.make_params
    # save_old, grad_lim, edge, node_res, qold_prim, sweep_prep, fill, sweeps, res_final
    assert bench.nc_kernels(p(flux="ausm", limiter="vkn", time="lusgs")) == 9
    # save_old, grad_lim, edge, node_res, sweep_prep, two fills, sweeps, res_final
    assert bench.nc_kernels(p(flux="ausm", limiter="vkn", time="lusgs", precision="mixed_sweep")) == 9
    assert bench.nc_kernels(p(flux="ausm", limiter="vkn", time="rk3")) == 5
    # the wall cells' partials are a launch of their own below two blocks of 256 cells per SM
    for sms in (100, 152):
        assert bench.cc_kernels(p(grad="gg"), (2 * sms - 1) * 256, sms) == 10
        assert bench.cc_kernels(p(grad="gg"), (2 * sms - 1) * 256 + 1, sms) == 9


def test_printed_line_is_short_and_whole(bench):
    """Every key of the contract, in a line that the tail of a log (3 000
    characters) holds, whatever the details come to."""
    deep = {"value": 123.456, "unit": bench.UNIT, "seconds": 12.3, "text": "x" * 4000}
    out = {"metric": bench.METRIC, "value": 73.8, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 7.1, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "gpu_library": "unsflow_gpu",
           "dtype": "f64", "data": "synthetic: seeded analytic-airfoil O-mesh, uniform freestream start", "gpu_launches": 180,
           "config": {"workload": max((w["desc"] for w in bench.WORKLOADS.values()), key=len), "units": 525312,
                      "global_batch": 525312, "seq_len": 1, "parallelism": "replicas x1", "l2": "x" * 100, "setup_s": 1.0,
                      "block_sizes": {"face": 256, "vertex": 256, "cell_grad": 128}},
           "e2e": {"value": 71.23456789, "unit": bench.UNIT, "h2d_bytes_per_step": 16809984, "d2h_bytes_per_step": 16810008,
                   "path": "x" * 200},
           "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 12},
           "roofline": {"bound": "hbm", "kernel": "lusgs_sweeps", "achieved": 58.2, "peak": 6796.9, "unit": "GB/s",
                        "frac": 0.0086, "traffic": 414432140, "duration_ms": 6.1, "latency_floor": deep},
           "kernels": deep, "cpu_baseline": dict(deep, cores=1, kind="port"), "parity": {"pass": True, "iterations": 50},
           "time_to_1e-8": {"mesh": "x", "fp64": deep, "mixed_sweep": deep},
           "configs": dict({k: deep for k, _ in bench.CONFIG_RUNS}, fp64_fma={"2": deep, "3_fp64": {"error": "x" * 400}})}
    line = bench.headline(out)
    assert len(json.dumps(line)) < 3000
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
              "dtype", "data", "gpu_launches"):
        assert line[k] == out[k]
    assert line["e2e"] == {"value": 71.235, "unit": bench.UNIT, "h2d_bytes_per_step": 16809984, "d2h_bytes_per_step": 16810008}
    assert line["clocks"] == out["clocks"] and line["config"]["units"] == 525312
    assert line["configs"] == {k: 123.456 for k, _ in bench.CONFIG_RUNS}
    assert line["time_to_1e-8_s"] == {"fp64": 12.3, "mixed_sweep": 12.3}
