"""The X pass kernels at every half-line length they are built for.

One grid nx x 18 x 16 per length (288 lines: a ragged last CTA for most line
counts), the OTC core with periodic and with zero-outside derivatives and the
OT core (whose X2 and X3 stop early, with the penalty in X3); poten's fields
(poten.f90:27-126, term_alfa.f90:157-236) must equal the FP64 oracle's.

Tolerances (relative to each field's maximum), as for the Y and Z passes: 25
roundings of a transform pair, times 10 for a gradient: FP64 1e-12, double-
float 1e-10, FP32 1e-4.  pot4 and U_alpha take ten times that (a second
derivative, and the penalty's rounding, 1.1e-16 x 3.2e4 K of some 10 K).
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu

HALF = [8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100,
        108, 120, 128, 135, 144, 150, 160, 162]
TOL = {"fp64": 1e-12, "dfloat": 1e-10, "fp32": 1e-4}
PREC = {"fp64": _abi.EP_FP64, "dfloat": _abi.EP_DFLOAT, "fp32": _abi.EP_FP32}
FIELDS = {"OTC": ("dencg", "delj4", "falfs", "intxalf", "intyalf", "intzalf", "ualphas", "pot4"),
          "OT ": ("dencg", "delj4", "pot4")}


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


@pytest.mark.parametrize("n2", HALF)
def test_poten_matches_the_oracle(oracle, n2):
    dims, h = (2 * n2, 18, 16), 0.8
    psi = _psi(dims, n2)
    for core, icon in (("OTC", _abi.EP_ICON_PERIODIC), ("OTC", _abi.EP_ICON_ZERO_OUTSIDE), ("OT ", _abi.EP_ICON_PERIODIC)):
        kw = dict(nx=dims[0], ny=dims[1], nz=dims[2], xmax=dims[0] * h / 2, ymax=dims[1] * h / 2, zmax=dims[2] * h / 2,
                  core=core, icon=icon, n4=100.0)
        with oracle.OracleSolver(ep.make_config(precision=_abi.EP_FP64, **kw)) as o:
            o.upload_psi(psi)
            o.poten()
            want = {f: o.field(f) for f in FIELDS[core]}
        for name, prec in PREC.items():
            with ep.Solver(ep.make_config(precision=prec, **kw)) as s:
                s.upload_psi(psi)
                s.poten()
                for f in FIELDS[core]:
                    err = np.max(np.abs(s.field(f) - want[f])) / np.max(np.abs(want[f]))
                    lim = TOL[name] * (10 if f in ("pot4", "ualphas") else 1)
                    assert err < lim, (name, dims, core, icon, f, err)
