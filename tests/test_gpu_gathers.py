"""The per-row gathers on sensors off the range-cell rule (a pulse table whose
taps are not one output range apart): the tensor-core gather with its split hot
tiles, and the CUDA-core one (RTACX_FLAG_SIMT_GATHER) in its three tile shapes,
each against the FP64 oracle at the plain form's 1e-5 relative L2, and against
each other at half of it. That the gathers ran is read from the stage times:
they alone have windows."""
import numpy as np
import pytest

from rtac_simulation_gb300 import _lib
from rtac_simulation_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

from helpers_gpu import gpu_reduce, make_context, rel_l2  # noqa: E402

TOL = 1e-5


def gathered(wk, flags=0):
    ctx = make_context(wk, flags=flags)
    ctx.set_tracing(True)
    if wk.echo:
        ctx.set_echo_model(wk.echo["carrier_hz"], wk.echo["flags"])
    out = gpu_reduce(ctx, wk.samples, wk.out_shape)
    return out, ctx.stage_times()["windows"] > 0.0


@pytest.mark.parametrize("duration", [0.5, 1.01])
@pytest.mark.parametrize("maker", [
    lambda: wl.oculus_2d(n_samples=1 << 18),                                        # 16 x 64 tiles, a seafloor
    lambda: wl.oculus_2d(n_samples=1 << 16, n_bearings=640),                        # 16 x 128
    lambda: wl.oculus_2d(n_samples=1 << 14, n_bearings=100, n_ranges=300),
    lambda: wl.precision_2d(n_samples=1 << 14, n_ranges=4096),                      # 32 x 128, every bearing
    lambda: wl.stress_2d(n_samples=1 << 18, n_ranges=2048),                         # half of it in hot tiles
])
def test_gathers_off_the_cell_rule_match_fp64_oracle(oracle, maker, duration):
    wk = maker()
    wk.sensor["pulse_duration"] = float(np.float32(duration * wk.sensor["pulse_duration"]))
    tc, tc_rows = gathered(wk)
    simt, simt_rows = gathered(wk, _lib.RTACX_FLAG_SIMT_GATHER)
    assert tc_rows and simt_rows
    samples = oracle.apply_echo(wk.samples, wk.sensor, wk.echo) if wk.echo else wk.samples
    want = oracle.reduce(samples, wk.sensor)
    assert np.isfinite(tc).all()
    assert rel_l2(tc, want) <= TOL, rel_l2(tc, want)
    assert rel_l2(simt, want) <= TOL, rel_l2(simt, want)
    assert rel_l2(tc, simt) <= 0.5 * TOL, rel_l2(tc, simt)


def test_sensors_on_the_cell_rule_do_not_gather():
    for maker in (lambda: wl.oculus_2d(n_samples=1 << 14), lambda: wl.oculus_reference_2d()):
        assert not gathered(maker())[1]
