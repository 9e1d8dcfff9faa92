"""ep_convolve_noalloc takes a d_out at any double's address (a slice of a
host's buffer), on grids whose last X pass is a per-length kernel and on one
whose is the general engine's, and writes nothing outside it; pointers that its
loads cannot take are refused on the host, before any device work."""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 32, 32), (30, 54, 64), (4, 16, 16), (320, 16, 16)])
def test_output_at_an_odd_double(dims):
    torch = pytest.importorskip("torch")
    build()
    f = ep.load_library()[1]["convolve_noalloc"]
    nx, ny, nz = dims
    n = nx * ny * nz
    a = torch.rand(nz, ny, nx, dtype=torch.float64, device="cuda")
    ker = torch.ones(nz, ny, nx // 2 + 1, dtype=torch.float64, device="cuda")
    buf = torch.full((n + 3,), -7.0, dtype=torch.float64, device="cuda")
    assert buf.data_ptr() % 16 == 0
    out = buf[1:n + 1]
    assert f(a.data_ptr(), ker.data_ptr(), out.data_ptr(), nx, ny, nz,
             torch.cuda.current_stream().cuda_stream) == _abi.EP_OK
    # the identity: 25 roundings of a transform pair, with a margin of about 40
    assert float((out - a.reshape(-1)).abs().max()) < 1e-13
    assert np.array_equal(buf[[0, n + 1, n + 2]].cpu().numpy(), [-7.0] * 3)


def test_refuses_addresses_its_loads_cannot_take():
    torch = pytest.importorskip("torch")
    build()
    f = ep.load_library()[1]["convolve_noalloc"]
    n = 16 * 16 * 16
    buf = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
    p = buf.data_ptr()
    st = torch.cuda.current_stream().cuda_stream
    assert f(p + 8, p, p, 16, 16, 16, st) == _abi.EP_ERR_INVALID_ARG
    assert f(p, p + 4, p, 16, 16, 16, st) == _abi.EP_ERR_INVALID_ARG
    assert f(p, p, p + 4, 16, 16, 16, st) == _abi.EP_ERR_INVALID_ARG
    torch.cuda.synchronize()
    assert torch.all(buf == 0)
