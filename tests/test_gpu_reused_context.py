"""Jobs one after another on one context.

After reset() a job must be the one a new context runs: the same bits, forty
times over, in every arithmetic, with a moving impurity whose internal
variables evolve in a potential (a 1000 K core) that makes the method amplify
its modifiers.  Without reset() the previous job's modifiers are carried, and
where they have grown beyond use the next start must drop them: the job's
internal variables stay near norm 1 (the first job's deviate by 1e-3; 0.1 is
the bound here, the NaN came from 1.5 and beyond) and nothing is raised.
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
DT = 0.5e-3 / ep.KTOPS


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build()


def _solver(prec):
    dims, h = (32, 32, 40), 1.0
    cfg = ep.make_config(nx=32, ny=32, nz=40, xmax=16.0, ymax=16.0, zmax=20.0, icon=_abi.EP_ICON_PERIODIC, core="OTC",
                         n4=300.0, impurity=_abi.EP_IMPURITY_MOVING, time_mode=_abi.EP_REAL_TIME, renormalize=0,
                         mimpur=40.0, fix_lambda=0, als_p=50.0, precision=prec)
    s = ep.Solver(cfg)
    s.set_impurity_potentials(ep.morse(10.0, 4.5, 1.2, 3.0, 1000.0), ep.morse(6.0, 5.0, 1.1, 3.0, 1000.0),
                              ep.morse(12.0, 4.0, 1.1))
    psi = ep.woods_saxon_psi(*dims, 16.0, 16.0, 20.0, 300.0, seed=5)
    return s, psi


def _job(s, psi):
    iv = np.zeros(10, dtype=np.complex128)
    iv[0], iv[3], iv[4] = 0.6, 0.64j, 0.48
    s.set_impurity(rimp=(0.0, 0.0, 0.3), vimp=(0.0, 0.0, 3.8), invar=iv)
    s.start(psi)
    for _ in range(4):
        s.steprk(DT)
    s.run(12, DT)
    s.poten()
    return dict(s.impurity(), psi=s.psi(), pc=s.cfield("pc"), energy=np.array(list(s.energy().values())))


@pytest.mark.parametrize("prec", [_abi.EP_FP64, _abi.EP_FP32, _abi.EP_DFLOAT], ids=["fp64", "fp32", "dfloat"])
def test_a_reset_context_repeats_the_first_job(prec):
    s, psi = _solver(prec)
    with s:
        first = _job(s, psi)
        for k in range(40):
            s.reset()
            again = _job(s, psi)
            for name in first:
                assert np.array_equal(first[name], again[name]), (k, name)


def test_lost_internal_variables_are_not_handed_on():
    s, psi = _solver(_abi.EP_FP64)
    with s:
        for k in range(40):
            got = _job(s, psi)
            assert abs(np.sum(np.abs(got["invar"]) ** 2) - 1.0) < 0.1, k
