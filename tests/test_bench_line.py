"""The bench's launch counts per iteration, against the launch sequences in the
sources (CPU)."""
import importlib.util
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
