"""run() skips, in all but its last step, the fields that only energy() and
the downloads read; what it leaves behind must be what the same number of
steppc() calls leaves, bit for bit: every field, the state, the energies, the
force and the moments (the stored values come from the same arithmetic, so no
tolerance applies)."""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
FIELDS = ["den", "pot4", "uimp", "dencg", "delj4", "dxden", "dyden", "dzden", "falfs", "intxalf", "intyalf", "intzalf",
          "ualphas", "vpi", "delta"]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build()


def _solver(prec, kind):
    dims, h = (32, 30, 36), 0.8
    kw = dict(nx=dims[0], ny=dims[1], nz=dims[2], xmax=dims[0] * h / 2, ymax=dims[1] * h / 2, zmax=dims[2] * h / 2,
              icon=_abi.EP_ICON_PERIODIC, core="OTC", n4=60.0, precision=prec)
    if kind == "fixed":
        kw.update(impurity=_abi.EP_IMPURITY_FIXED)
    else:
        kw.update(impurity=_abi.EP_IMPURITY_MOVING, mimpur=40.0, time_mode=_abi.EP_REAL_TIME, renormalize=0,
                  fix_lambda=1 if kind == "frozen" else 0, als_p=5.0)
    s = ep.Solver(ep.make_config(**kw))
    pot = ep.morse(10.0, 4.5, 1.2, 3.0, 500.0)
    s.set_impurity_potentials(pot, ep.morse(6.0, 5.0, 1.1, 3.0, 500.0), ep.morse(12.0, 4.0, 1.1))
    iv = np.zeros(10, dtype=np.complex128)
    iv[0], iv[3] = 0.6, 0.8j
    s.set_impurity(rimp=(0.2, -0.1, 0.3), vimp=(0.0, 0.0, 0.5), invar=iv)
    s.start(ep.woods_saxon_psi(*dims, kw["xmax"], kw["ymax"], kw["zmax"], 60.0, seed=2))
    for _ in range(3):
        s.steprk(2e-5)
    return s


def _left(s):
    out = {f: s.field(f) for f in FIELDS}
    out["psi"] = s.psi()
    out["force"] = s.forceimp()
    out["moments"] = s.impurity_moments()
    out["energy"] = np.array(list(s.energy().values()))
    out.update(s.impurity())
    return out


@pytest.mark.parametrize("kind", ["fixed", "frozen", "moving"])
@pytest.mark.parametrize("prec", [_abi.EP_FP64, _abi.EP_FP32, _abi.EP_DFLOAT], ids=["fp64", "fp32", "dfloat"])
@pytest.mark.parametrize("wait", [False, True])
def test_run_leaves_what_steppc_leaves(prec, kind, wait):
    with _solver(prec, kind) as a, _solver(prec, kind) as b:
        for n in (1, 5, 3):  # a second and third call start from replayed graphs
            a.run(n, 2e-5, wait=wait)
            for _ in range(n):
                b.steppc(2e-5, wait=False)
            x, y = _left(a), _left(b)
            for k in x:
                assert np.array_equal(x[k], y[k]), (kind, n, k)
