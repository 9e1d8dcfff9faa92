"""The impurity field, its moments and the energy integrals on grids whose
columns, rows and chunks do not fill the launch (a partial last group of 32
columns, row chunks that split unevenly, fewer rows than a block's warps can
share), for both boundary modes, with a P state of two channels and an
excluded core, against the FP64 oracle.

Tolerances: sums and fields carry the fields' own rounding -- FP64 1e-11 (the
parity gate), double-float the same, FP32 2e-5 of the largest entry.
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
PREC = {"fp64": (_abi.EP_FP64, 1e-11), "dfloat": (_abi.EP_DFLOAT, 1e-11), "fp32": (_abi.EP_FP32, 2e-5)}


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build()


@pytest.mark.parametrize("plus", ["morse", "ion"])
@pytest.mark.parametrize("icon", [_abi.EP_ICON_PERIODIC, _abi.EP_ICON_ZERO_OUTSIDE])
@pytest.mark.parametrize("dims", [(16, 18, 16), (30, 54, 18), (48, 20, 50), (100, 96, 16)])
def test_fields_moments_and_energies(oracle, dims, icon, plus):
    nx, ny, nz = dims
    h = 0.8
    kw = dict(nx=nx, ny=ny, nz=nz, xmax=nx * h / 2, ymax=ny * h / 2, zmax=nz * h / 2, core="OTC", icon=icon, n4=80.0,
              impurity=_abi.EP_IMPURITY_MOVING, mimpur=40.0, als_p=20.0,
              z_exciplex_exclusion=0.0 if plus == "morse" else 1.5)
    psi = ep.woods_saxon_psi(nx, ny, nz, kw["xmax"], kw["ymax"], kw["zmax"], 80.0, seed=7)
    iv = np.zeros(10, dtype=np.complex128)
    iv[0], iv[3], iv[4] = 0.6, 0.64j, 0.48

    def fill(s):
        s.set_impurity_potentials(ep.morse(10.0, 4.5, 1.2, 2.0, 800.0), ep.morse(6.0, 5.0, 1.1, 2.0, 800.0),
                                  ep.morse(12.0, 4.0, 1.1, 2.5, 500.0) if plus == "morse" else ep.koutselos("K", 2.0, 900.0))
        s.set_impurity(rimp=(0.31, -0.23, 0.57), vimp=(0.1, 0.2, 0.3), invar=iv)
        s.start(psi)
        return dict(uimp=s.field("uimp"), vpi=s.field("vpi"), delta=s.field("delta"), force=s.forceimp(),
                    potinvar=s.potinvar(), energy=s.energy())

    with oracle.OracleSolver(ep.make_config(precision=_abi.EP_FP64, **kw)) as o:
        want = fill(o)
    for name, (prec, tol) in PREC.items():
        with ep.Solver(ep.make_config(precision=prec, **kw)) as s:
            got = fill(s)
        for k in ("uimp", "vpi", "delta", "force", "potinvar"):
            err = np.max(np.abs(got[k] - want[k])) / np.max(np.abs(want[k]))
            # the force is a sum that cancels: held to the size of its terms
            lim = tol * (50.0 if k == "force" else 1.0)
            assert err < lim, (name, dims, k, err)
        scale = max(abs(v) for v in want["energy"].values())
        for k, v in want["energy"].items():
            assert abs(got["energy"][k] - v) <= tol * max(abs(v), 1e-3 * scale), (name, dims, k, got["energy"][k], v)
