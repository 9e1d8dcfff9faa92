"""Impurity tables replaced on a live context are the ones that the next
potenimp() reads: nothing lies between the two calls, so the kernel must be
ordered behind the upload.  Each field must be, bit for bit, that of a new
context with the same tables, in both states and all arithmetics."""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
MORSE = [(10.0, 4.5, 1.2, 3.0, 1000.0), (6.0, 5.0, 1.1, 2.5, 700.0)]


def _solver(prec, state):
    cfg = ep.make_config(nx=64, ny=32, nz=16, xmax=12.8, ymax=6.4, zmax=3.2, core="OTC", n4=100.0, state=state,
                         icon=_abi.EP_ICON_PERIODIC, precision=prec, impurity=_abi.EP_IMPURITY_FIXED)
    s = ep.Solver(cfg)
    iv = np.zeros(10, dtype=np.complex128)
    iv[0], iv[3] = 0.6, 0.8j
    s.set_impurity(rimp=(0.2, -0.1, 0.3), invar=iv)
    return s


def _field(s, state, k):
    a, b = ep.morse(*MORSE[k]), ep.morse(*MORSE[1 - k])
    if state == _abi.EP_STATE_D:
        s.set_impurity_potentials_d(a, b, ep.morse(8.0, 4.8, 1.15, 2.8, 900.0 + k))
    else:
        s.set_impurity_potentials(a, b)
    s.potenimp()
    return s.field("uimp")


@pytest.mark.parametrize("state", [_abi.EP_STATE_P, _abi.EP_STATE_D], ids=["P", "D"])
@pytest.mark.parametrize("prec", [_abi.EP_FP64, _abi.EP_FP32, _abi.EP_DFLOAT], ids=["fp64", "fp32", "dfloat"])
def test_the_next_field_is_of_the_new_tables(prec, state):
    build()
    want = []
    for k in (0, 1):
        with _solver(prec, state) as s:
            _field(s, state, k)
            s.synchronize()
            s.potenimp()
            want.append(s.field("uimp"))
    assert not np.array_equal(*want)
    with _solver(prec, state) as s:
        for i in range(30):
            assert np.array_equal(_field(s, state, i % 2), want[i % 2]), i
