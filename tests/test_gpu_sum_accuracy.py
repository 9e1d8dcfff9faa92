"""The sums of double-float and FP32 fields (energy integrals, the force)
against sums of the same fields in extended precision.

Tolerances, relative to the sum of the terms' magnitudes: products round by
2^-46 and threads' pairs by 2^-49 at random over more than 1e5 points (below
1e-16), a block's FP64 tree by eight times 2^-53 at random over the blocks, the
result once: 1e-15 holds them with a margin of about five.  The solid penalty's
exponential is good to 2^-37.  FP32 fields' force is summed in FP32 (its products
round by 2^-24 at random): 1e-7.
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.mark.parametrize("prec", [_abi.EP_DFLOAT, _abi.EP_FP32], ids=["dfloat", "fp32"])
@pytest.mark.parametrize("dims,h", [((64, 64, 64), 0.8), ((60, 72, 80), 0.5), ((50, 48, 64), 0.8)])
def test_sums_of_the_fields(dims, h, prec):
    build()
    nx, ny, nz = dims
    cfg = ep.make_config(nx=nx, ny=ny, nz=nz, xmax=nx * h / 2, ymax=ny * h / 2, zmax=nz * h / 2, core="OTC", n4=300.0,
                         icon=_abi.EP_ICON_PERIODIC, impurity=_abi.EP_IMPURITY_MOVING, mimpur=40.0, precision=prec)
    psi = ep.woods_saxon_psi(nx, ny, nz, cfg.xmax, cfg.ymax, cfg.zmax, 300.0, seed=3)
    with ep.Solver(cfg) as s:
        s.set_impurity_potentials(ep.morse(10.0, 4.5, 1.2), plus=ep.morse(12.0, 4.0, 1.1))
        s.set_impurity(rimp=(0.31, -0.23, 0.57), invar=np.zeros(10, dtype=np.complex128))
        s.start(psi)
        e, F, dv = s.energy(), s.forceimp(), L(s.dxyz)
        f = {k: s.field(k).astype(L) for k in ("den", "uimp", "dencg", "delj4", "dxden", "dyden", "dzden")}
    den, cg = f["den"], f["dencg"]
    t = 2 * L(cfg.beta) * (den - L(cfg.den_m))
    penalty = den * 2 * np.exp(t) / (1 + np.exp(t))
    checks = {"n4": (e["n4"], [den * dv], 1e-15),
              "eHeX": (e["eHeX"], [den * f["uimp"] * dv], 1e-15),
              "elj4": (e["elj4"], [den * f["delj4"] * dv / 2], 1e-15),
              "ecor4": (e["ecor4"], [den * cg**2 * (L(cfg.cp4) / 2) * dv, den * cg**3 * (L(cfg.cpp4) / 3) * dv], 1e-15),
              "esolid": (e["esolid"], [L(cfg.C) * penalty * dv], 2.0 ** -37)}
    for i, k in enumerate(("dxden", "dyden", "dzden")):
        checks[f"force {k}"] = (F[i], [-f[k] * f["uimp"] * dv], 1e-15 if prec == _abi.EP_DFLOAT else 1e-7)
    for name, (got, terms, tol) in checks.items():
        want, size = sum(v.sum() for v in terms), sum(abs(v).sum() for v in terms)
        assert abs(L(got) - want) <= tol * size, (name, float(abs(L(got) - want) / size))
