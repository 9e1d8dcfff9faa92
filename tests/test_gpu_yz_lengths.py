"""The Y and Z pass kernels at every length they are built for.

Each grid 16 x n x m takes a pair of lengths, so that every length runs as a
Y axis (in-place passes, forward and inverse) and as a Z axis (convolutions
with one and with three form-factor tables), with a ragged last tile of lines
(9 n and 9 m lines are no multiple of the tiles).  The convolved fields of
poten (poten.f90:27-50, term_alfa.f90:157-181) must equal the FP64 oracle's.

Tolerances (relative to each field's maximum): a transform pair of 2^a 3^b 5^c
points rounds about log2(N) times, 25 units for these grids, times 10 for the
gradient in the alpha_s integrals: FP64 1.1e-16 -> 1e-12 with a margin of
about 40; double-float 2^-44 -> 1e-10; FP32 6e-8 -> 1e-4.
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu

LENGTHS = [16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 162,
           180, 192, 200, 216, 240, 256, 270, 288, 300, 320, 324]
TOL = {"fp64": 1e-12, "dfloat": 1e-10, "fp32": 1e-4}
PREC = {"fp64": _abi.EP_FP64, "dfloat": _abi.EP_DFLOAT, "fp32": _abi.EP_FP32}
FIELDS = ("dencg", "delj4", "falfs", "intxalf", "intyalf", "intzalf")


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build()


def _psi(dims, seed):
    """sqrt of 0.02 A^-3 modulated by a few plane waves along each axis and 1 % noise."""
    rng = np.random.default_rng(seed)
    rho = np.full(dims, 0.02)
    for axis, n in enumerate(dims):
        shape = [1, 1, 1]
        shape[axis] = n
        x = 2 * np.pi * np.arange(n).reshape(shape) / n
        for k in (1, 2, n // 3):
            rho = rho * (1 + 0.05 * np.cos(k * x + rng.uniform(0, 6)))
    rho = rho * (1 + 0.01 * rng.random(dims))
    return np.asfortranarray(np.sqrt(rho).astype(np.complex128))


@pytest.mark.parametrize("n", LENGTHS)
def test_convolved_fields_match_the_oracle(oracle, n):
    m = LENGTHS[(LENGTHS.index(n) + 17) % len(LENGTHS)]
    dims, h = (16, n, m), 0.8
    kw = dict(nx=dims[0], ny=n, nz=m, xmax=dims[0] * h / 2, ymax=n * h / 2, zmax=m * h / 2, core="OTC",
              icon=_abi.EP_ICON_PERIODIC, n4=100.0)
    psi = _psi(dims, n)
    with oracle.OracleSolver(ep.make_config(precision=_abi.EP_FP64, **kw)) as o:
        o.upload_psi(psi)
        o.poten()
        want = {f: o.field(f) for f in FIELDS}
    for name, prec in PREC.items():
        with ep.Solver(ep.make_config(precision=prec, **kw)) as s:
            s.upload_psi(psi)
            s.poten()
            for f in FIELDS:
                err = np.max(np.abs(s.field(f) - want[f])) / np.max(np.abs(want[f]))
                assert err < TOL[name], (name, dims, f, err)
