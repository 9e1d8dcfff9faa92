"""The impurity field beside a cut-off core, where update()'s parabola spans the
jump: Delta and V_Pi against the parabola through the three table points
evaluated in extended precision at the same r.

Tolerance: the slope there is jump / (2 h) (2 h the parabola's span) and r
and the table index carry two roundings of r: |dV| <= 2 u r jump / h, plus four
roundings of the field's values; twice that is the bound.  Coefficients about
r = 0 miss it by jump / h^2 r^2 u / (r jump / h u) = r / h, several hundred.
"""
import numpy as np
import pytest

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi
from eff_pot_gb300.build import build

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.mark.parametrize("prec,u", [(_abi.EP_FP64, 2.0 ** -53), (_abi.EP_DFLOAT, 2.0 ** -48)], ids=["fp64", "dfloat"])
@pytest.mark.parametrize("dims,rc", [((64, 64, 80), 3.0), ((30, 54, 18), 2.0), ((100, 16, 20), 4.0)])
def test_field_beside_the_core(dims, rc, prec, u):
    build()
    nx, ny, nz = dims
    h, umax = 0.5, 1000.0
    cfg = ep.make_config(nx=nx, ny=ny, nz=nz, xmax=nx * h / 2, ymax=ny * h / 2, zmax=nz * h / 2, core="OTC", n4=100.0,
                         icon=_abi.EP_ICON_PERIODIC, precision=prec, impurity=_abi.EP_IMPURITY_FIXED)
    pi, sg = ep.morse(10.0, 4.5, 1.2, rc, umax), ep.morse(6.0, 5.0, 1.1, rc, 0.4 * umax)
    rimp = np.array([0.31, -0.23, 0.57])
    with ep.Solver(cfg) as s:
        s.set_impurity_potentials(pi, sg)
        s.set_impurity(rimp=rimp, invar=np.zeros(10, dtype=np.complex128))
        s.potenimp()
        got = {k: s.field(k) for k in ("vpi", "delta")}
        x, y, z = (a - b for a, b in zip(s.axes(), rimp))
    r2 = (x * x)[:, None, None] + ((y * y)[None, :, None] + (z * z)[None, None, :])
    r = np.sqrt(r2)
    npot = 100 * max(dims) + 1
    dr = 4.0 * max(cfg.xmax, cfg.ymax, cfg.zmax) / (npot - 1)
    i0 = np.clip((1.5 + r / dr).astype(int), 1, npot)
    at = np.arange(npot) * dr
    tp = ep.potential_values(pi, at)
    td = ep.potential_values(sg, at) - tp
    for k, t in (("vpi", tp), ("delta", td)):
        f = np.concatenate([t[:1], t, t[-1:]]).astype(L)
        d = r.astype(L) - (i0 - 1) * L(dr)
        fm, f0, fp = f[i0 - 1], f[i0], f[i0 + 1]
        want = f0 + d * ((fp - fm) / 2 + (fp - 2 * f0 + fm) / 2 * (d / L(dr))) / L(dr)
        lim = 2 * (2 * 2.0 ** -53 * r * (abs(fp - f0) + abs(f0 - fm)) / dr + 4 * u * abs(want))
        if k == "delta":
            want, lim = want / r2, lim / r2
        far = r > 2e-3
        jump = (abs(fp - f0) + abs(f0 - fm)) > 100.0
        assert np.any(jump & far)
        assert np.all((abs(got[k] - want) <= lim)[far]), (k, float(np.max((abs(got[k] - want) / lim)[far])))
