"""ep_convolve_noalloc on axes of every kind it dispatches: per-length kernels
on all axes, the general engine on one (X, Y or Z) or all of them (odd axes,
2 points, 3 x 3 x 5 points), ragged tiles.  Against numpy's FFT in FP64 with a
random kernel table; 25 roundings of a transform pair, 1.1e-16 each, with a
margin of about 40: 1e-13 of the result's maximum."""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 32, 32), (16, 18, 20), (54, 30, 30), (4, 16, 16), (16, 45, 16), (16, 16, 27),
                                  (2, 3, 5), (250, 9, 15), (20, 96, 48), (30, 54, 64)])
def test_matches_numpy(dims):
    torch = pytest.importorskip("torch")
    build()
    f = ep.load_library()[1]["convolve_noalloc"]
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + ny + nz)
    a = rng.random((nz, ny, nx))
    ker = rng.random((nz, ny, nx // 2 + 1))
    # a table of a real convolution: equal at k and -k on the planes kx = 0 and nx/2
    for p in (0, nx // 2):
        m = ker[:, :, p]
        ker[:, :, p] = 0.5 * (m + np.roll(m[::-1, ::-1], (1, 1), (0, 1)))
    want = np.fft.irfftn(np.fft.rfftn(a) * ker, s=a.shape, axes=(0, 1, 2))
    d_a, d_k = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, ker))
    out = torch.empty_like(d_a)
    for _ in range(2):
        out.fill_(float("nan"))
        assert f(d_a.data_ptr(), d_k.data_ptr(), out.data_ptr(), nx, ny, nz,
                 torch.cuda.current_stream().cuda_stream) == _abi.EP_OK
        got = out.cpu().numpy()
        assert np.max(np.abs(got - want)) < 1e-13 * np.max(np.abs(want))
