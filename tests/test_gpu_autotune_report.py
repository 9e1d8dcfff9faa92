"""The autotuner reports launch shapes for the axes that have them only: one
longer than every per-length kernel (360 points) does, the others are named
as their length's own."""
import re

import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,shaped", [((48, 48, 48), ""), ((16, 16, 360), "Z"), ((16, 360, 16), "Y"),
                                         ((360, 16, 16), "X1..X4")])
def test_report_names_the_shapes_in_use(dims, shaped):
    build()
    nx, ny, nz = dims
    cfg = ep.make_config(nx=nx, ny=ny, nz=nz, xmax=0.4 * nx, ymax=0.4 * ny, zmax=0.4 * nz, core="OTC", n4=50.0,
                         icon=_abi.EP_ICON_PERIODIC, precision=_abi.EP_FP32)
    with ep.Solver(cfg) as s:
        s.start(ep.woods_saxon_psi(nx, ny, nz, cfg.xmax, cfg.ymax, cfg.zmax, 50.0, seed=1))
        rep = s.autotune()
    parts = dict(re.findall(r"(X1\.\.X4|Y|Z) ([^,]+)", rep))
    assert set(parts) == {"X1..X4", "Y", "Z"}, rep
    for axis, text in parts.items():
        assert (re.match(r"\d+x\d+", text) is not None) == (axis == shaped), rep
