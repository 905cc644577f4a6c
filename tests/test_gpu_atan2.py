"""The echo epilogue's bearing, atan2(-ly, lx) of the hit's direction: over all
octants, their edges, and magnitudes outside the polynomial's range (which the
library function takes), against numpy in float64. Tolerance: 4 units of
2^-24 pi (the library's own bound is 3 ulp)."""
import numpy as np
import pytest

from rtac_simulation_gb300 import _lib
from rtac_simulation_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

from helpers_gpu import make_context  # noqa: E402


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 4097, 300001])
def test_bearings_over_all_octants(n, offset):
    rng = np.random.default_rng(n)
    a = rng.uniform(-np.pi, np.pi, n)
    r = 10.0 ** rng.uniform(-34.0, 34.0, n)
    x, y = (r * np.cos(a)).astype(np.float32), (r * np.sin(a)).astype(np.float32)
    edge = np.array([[0, 0], [1, 0], [-1, 0], [0, 1], [0, -1], [1, 1], [-1, 1], [1, -1], [-1, -1], [1e-38, 1e38],
                     [-0.0, 1], [-0.0, -0.0], [1e-44, 1e-44], [-3e38, 1]], np.float32)[:n]
    x[:len(edge)], y[:len(edge)] = edge[:, 0], edge[:, 1]
    hits = np.zeros((n, 6), np.float32)
    hits[:, 0], hits[:, 2] = 1.0, 3.0
    hits[:, 3], hits[:, 4] = x, y
    wk = wl.oculus_reference_2d(n_samples=16)
    ctx = make_context(wk)
    ctx.configure_receiver(np.eye(3), None, carrier_hz=0.0, flags=0)
    buf = torch.zeros(hits.size + 4, device="cuda")
    buf[offset:offset + hits.size] = torch.from_numpy(hits.reshape(-1)).cuda()
    out = torch.empty((n, 4), device="cuda")
    ctx.make_samples(buf[offset:], n, out, stream=torch.cuda.current_stream())
    got = out.cpu().numpy()[:, 3].astype(np.float64)
    # the identity rotation's sums, in which a zero's sign is lost as in the kernel
    local = (hits[:, None, 3:6] * np.eye(3, dtype=np.float32)).sum(axis=2, dtype=np.float32)
    want = np.arctan2(-local[:, 1].astype(np.float64), local[:, 0].astype(np.float64))
    assert np.max(np.abs(got - want)) <= 4 * np.pi * 2.0 ** -24
