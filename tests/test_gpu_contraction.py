"""The precision form's split contraction on its own: samples on the grid's
nodes (so that the binned grid holds their values exactly) and one range tap of
1, which leave out(r, b) = sum_q G[r / 2][q] D[q][b], against float64. Sums over
a few and over the most grid bearings (K parts 1 to 16, both tile widths), a
column tile whose directivity is zero, and both operand types.

All terms of the real part are positive, so that truncation adds up. Tolerances:
no accumulator sums more than 2200 terms at 6e-9 each, 1.32e-5; a bf16 pair
holds 16 bits of either operand, 2^-16 for a product; an fp16 pair 22 bits and
the dropped product 2^-22, together below 2^-20."""
import numpy as np
import pytest

from rtac_simulation_gb300 import _lib
from rtac_simulation_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)


@pytest.mark.parametrize("fp16", [False, True])
@pytest.mark.parametrize("nR,nB,cells,zero", [
    (64, 64, 64, None), (512, 128, 512, None), (512, 200, 512, (64, 128)), (300, 500, 2000, None),
    (4096, 512, 2048, (0, 128)), (64, 64, 8192, None), (40, 70, 16384, (64, 70)),
])
def test_contraction_matches_float64(nR, nB, cells, zero, fp16):
    res, step, first = 1.0 / 64, 2.0 ** -14, -0.5
    ctx = _lib.Context(0)
    bearings = np.linspace(-0.4, 0.4, nB).astype(np.float32)
    ctx.configure_2d(**wl.sensor_2d(0.0, (nR - 1) * res, nR, 1500.0, np.ones(4, np.complex64), 4 * res,
                                    np.ones(9, np.float32), 0.5, bearings))
    g = torch.Generator(device="cuda").manual_seed(nR + nB + cells)
    u = lambda *shape: torch.rand(shape, generator=g, device="cuda") * 0.5 + 0.5  # noqa: E731
    D = torch.complex(u(cells, nB), -u(cells, nB))
    if zero:
        D[:, zero[0]:zero[1]] = 0
    ctx.configure_precision(directivity=D.cpu().numpy(), range_taps=np.ones((2, 1), np.complex64), tap_center=0,
                            grid_count=cells, grid_first=first, grid_last=first + (cells - 1) * step,
                            flags=_lib.RTACX_PRECISION_FP16_ROWSCALE if fp16 else 0)
    nodes = (nR - 1) // 2 + 1
    G = torch.complex(u(nodes, cells), u(nodes, cells))
    smp = torch.empty((nodes, cells, 4), device="cuda")
    smp[..., 0], smp[..., 1] = G.real, G.imag
    smp[..., 2] = (torch.arange(nodes, device="cuda") * (2 * res))[:, None]
    smp[..., 3] = first + torch.arange(cells, device="cuda") * step
    out = torch.full((nR, nB, 2), float("nan"), device="cuda")
    stream = torch.cuda.current_stream()
    ctx.reduce_precision(smp, nodes * cells, out, stream=stream)
    ctx.stream_status(stream)
    want = (G.to(torch.complex128) @ D.to(torch.complex128))[torch.arange(nR, device="cuda") // 2]
    got = torch.view_as_complex(out).to(torch.complex128)
    err = float((got.real - want.real).norm() / want.real.norm())
    print(f"{nR} x {nB}, {cells} grid bearings, {'fp16' if fp16 else 'bf16'}: {err:.2e}")
    assert err <= 1.32e-5 + (2.0 ** -20 if fp16 else 2.0 ** -16), err
    if zero:
        assert torch.count_nonzero(out[:, zero[0]:zero[1]]).item() == 0
