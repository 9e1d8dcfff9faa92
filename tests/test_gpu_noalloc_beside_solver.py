"""ep_convolve_noalloc and FP64 contexts in one process launch the same
kernels: a convolution must leave a context of the same axis lengths working
(poten's convolutions with two and three tables take twice its shared
memory), and after the first call a call of any other size must be capturable.
"""
import subprocess
import sys

import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [192, 200, 216, 240, 256])
def test_a_convolution_leaves_the_solver_working(n):
    torch = pytest.importorskip("torch")
    build()
    f = ep.load_library()[1]["convolve_noalloc"]
    cfg = ep.make_config(nx=16, ny=16, nz=n, xmax=6.4, ymax=6.4, zmax=0.4 * n, core="OTC", n4=50.0,
                         icon=_abi.EP_ICON_PERIODIC, precision=_abi.EP_FP64)
    psi = ep.woods_saxon_psi(16, 16, n, cfg.xmax, cfg.ymax, cfg.zmax, 50.0, seed=1)
    a = torch.rand(n, 16, 16, dtype=torch.float64, device="cuda")
    ker, out = torch.ones(n, 16, 9, dtype=torch.float64, device="cuda"), torch.empty_like(a)
    with ep.Solver(cfg) as s:
        s.upload_psi(psi)
        s.poten()
        want = s.field("pot4")
        assert f(a.data_ptr(), ker.data_ptr(), out.data_ptr(), 16, 16, n,
                 torch.cuda.current_stream().cuda_stream) == _abi.EP_OK
        s.poten()
        assert np.array_equal(s.field("pot4"), want)
    # the identity: 25 roundings of a transform pair, with a margin of about 40
    assert float((out - a).abs().max()) < 1e-13


CAPTURE = """
import torch, eff_pot_gb300 as ep
f = ep.load_library()[1]["convolve_noalloc"]
def call(nx, ny, nz):
    a = torch.rand(nz, ny, nx, dtype=torch.float64, device="cuda")
    k, o = torch.ones(nz, ny, nx // 2 + 1, dtype=torch.float64, device="cuda"), torch.zeros_like(a)
    return a, o, lambda: f(a.data_ptr(), k.data_ptr(), o.data_ptr(), nx, ny, nz, torch.cuda.current_stream().cuda_stream)
assert call(16, 16, 16)[2]() == 0
for dims in ((32, 24, 40), (10, 15, 192), (320, 16, 16)):
    a, o, run = call(*dims)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert run() == 0
    g.replay()
    torch.cuda.synchronize()
    assert float((o - a).abs().max()) < 1e-13, dims
print("captured")
"""


def test_a_call_of_another_size_can_be_captured():
    pytest.importorskip("torch")
    build()
    r = subprocess.run([sys.executable, "-c", CAPTURE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
