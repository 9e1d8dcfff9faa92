"""What run() leaves behind, over every way it replays its steps: single and
multi-step graphs, runs of whole rotation periods and others, with and without
statistics, the first call of a length and later ones, batches with and without
a moving impurity, the OTC and OT cores.  Each must be, bit for bit, what the same number of
steppc() calls on contexts of their own leaves (the stored values come from the
same arithmetic)."""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
FIELDS = ["den", "pot4", "uimp", "dencg", "delj4", "dxden", "dyden", "dzden", "falfs", "intxalf", "intyalf", "intzalf",
          "ualphas", "vpi", "delta"]
DT = 2e-5


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build()


def _config(kind, core, prec):
    kw = dict(nx=32, ny=30, nz=36, xmax=12.8, ymax=12.0, zmax=14.4, icon=_abi.EP_ICON_PERIODIC, core=core, n4=60.0,
              precision=prec)
    if kind == "fixed":
        kw.update(impurity=_abi.EP_IMPURITY_FIXED)
    else:
        kw.update(impurity=_abi.EP_IMPURITY_MOVING, mimpur=40.0, time_mode=_abi.EP_REAL_TIME, renormalize=0,
                  fix_lambda=1, als_p=5.0)
    return ep.make_config(**kw)


def _fill(s, seed):
    s.set_impurity_potentials(ep.morse(10.0, 4.5, 1.2, 3.0, 500.0), ep.morse(6.0, 5.0, 1.1, 3.0, 500.0),
                              ep.morse(12.0, 4.0, 1.1))
    iv = np.zeros(10, dtype=np.complex128)
    iv[0], iv[3] = 0.6, 0.8j
    s.set_impurity(rimp=(0.2, -0.1, 0.3), vimp=(0.0, 0.0, 0.5), invar=iv)
    s.start(ep.woods_saxon_psi(32, 30, 36, 12.8, 12.0, 14.4, 60.0, seed=seed))
    for _ in range(3):
        s.steprk(DT)


def _left(s):
    out = {f: s.field(f) for f in FIELDS}
    out.update(psi=s.psi(), pc=s.cfield("pc"), force=s.forceimp(), energy=np.array(list(s.energy().values())))
    out.update(s.impurity())
    return out


def _same(a, b, where):
    x, y = _left(a), _left(b)
    for k in x:
        assert np.array_equal(x[k], y[k]), (where, k)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("wait", [False, True])
@pytest.mark.parametrize("core,prec", [("OTC", _abi.EP_FP32), ("OT ", _abi.EP_FP32), ("OTC", _abi.EP_DFLOAT)])
def test_run_of_one_context(core, prec, wait, mode):
    cfg = _config("fixed", core, prec)
    with ep.Solver(cfg) as a, ep.Solver(cfg) as b:
        for s in (a, b):
            _fill(s, 2)
        a.step_graphs(mode)
        for n in (2, 10, 2, 21, 13, 10, 20, 1, 3):
            a.run(n, DT, wait=wait)
            for _ in range(n):
                b.steppc(DT, wait=False)
            _same(a, b, (mode, wait, n))


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("wait", [False, True])
@pytest.mark.parametrize("kinds", [("fixed", "fixed"), ("fixed", "frozen")])
def test_run_of_a_batch(kinds, wait, mode):
    cfgs = [_config(k, "OTC", _abi.EP_FP32) for k in kinds]
    batch, alone = ep.Batch(cfgs), [ep.Solver(c) for c in cfgs]
    try:
        for i in range(2):
            _fill(batch[i], 2 + i)
            _fill(alone[i], 2 + i)
        batch.step_graphs(mode)
        for n in (2, 12, 2, 20, 3):
            batch.run(n, DT, wait=wait)
            batch.synchronize()
            for i, s in enumerate(alone):
                for _ in range(n):
                    s.steppc(DT, wait=False)
                _same(batch[i], s, (kinds, mode, wait, n, i))
    finally:
        batch.close()
        for s in alone:
            s.close()
