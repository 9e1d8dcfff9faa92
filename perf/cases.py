"""The work that users have this framework do, as cases to be timed and compared.

Every case goes through the public entry points (Solver, Batch, and the C ABI
function ep_convolve_noalloc) in the way the driver, the benchmark and the
scan and real-time programs of this repository call them:

* convolve  one k-space convolution on device buffers of the caller;
* file      the per-density evaluation of the U*/U+ scan: upload, impurity
            field, mean field, energies;
* relax     an imaginary-time job on one droplet: upload, start-up,
            Runge-Kutta-Gill start, predictor-corrector steps (optionally a
            refinement in double-float at the end), energies and psi back;
* batch     the same job on many droplets advanced together;
* kick      a real-time job on a droplet with a moving impurity: upload,
            start-up, Runge-Kutta-Gill start, steps up to the first sample,
            mean field, energies, the impurity's place and velocity, psi.

Sizes and physical parameters are those of the benchmark's configurations and
of the tests; draw() varies them over every even 2^a 3^b 5^c grid between.
exact() restates the same physics in plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import eff_pot_gb300 as ep
from eff_pot_gb300 import _abi

DT = 1e-4                               # imaginary time, 1/K
DT_REAL = 0.5e-3 / ep.KTOPS             # real time, 0.5 fs
KICK = 50.0 * 1e10 / 1e12 * ep.KTOPS    # 50 m/s
MIMPUR = 40.0                           # impurity mass, u
RK_STEPS = 3                            # Runge-Kutta-Gill steps before the multistep method
PRECISION = {"fp64": _abi.EP_FP64, "fp32": _abi.EP_FP32, "dfloat": _abi.EP_DFLOAT}
MORSE = (10.0, 4.5, 1.2)                # the He-X pair potential (K, A, 1/A)
MORSE_SIGMA = (6.0, 5.0, 1.1)           # its sigma channel where the P state is anisotropic
CORE = (3.0, 1000.0)                    # r_cutoff and umax of both channels there (A, K)
MORSE_PLUS = (12.0, 4.0, 1.1)           # the ion's potential of U+
ENERGIES = ("etot", "etot4", "ekin4", "elj4", "ecor4", "ealphas", "esolid", "eimpu", "ekinx", "eHeX", "uplus",
            "eso", "n4")


def listed():
    return [
        # A host that may not allocate (it owns the memory pool, or captures a
        # graph) convolves one small density: latency and launches count.
        dict(name="convolve_32", kind="convolve", nx=32, ny=32, nz=32),
        # One density file of the reference's get_impurity_energy.sh loop, with
        # the driver's default zero-outside boundary.
        dict(name="file_64_fp64", kind="file", nx=64, ny=64, nz=64, h=0.8, n4=500.0, precision="fp64", core="OTC",
             periodic=False),
        # The small pure droplet (N = 500, h = 0.8 A) in bulk FP32 steps.
        dict(name="pure_64_fp32", kind="relax", nx=64, ny=64, nz=64, h=0.8, n4=500.0, precision="fp32", core="OTC",
             impurity=False, steps=100, refine=0),
        # The droplet + Morse impurity at 128^3 in each arithmetic: FP32 bulk
        # steps, the double-float path, the plain FP64 path.
        dict(name="drop_128_fp32", kind="relax", nx=128, ny=128, nz=128, h=0.4, n4=1000.0, precision="fp32",
             core="OTC", impurity=True, steps=42, refine=0),
        dict(name="drop_128_dfloat", kind="relax", nx=128, ny=128, nz=128, h=0.4, n4=1000.0, precision="dfloat",
             core="OTC", impurity=True, steps=16, refine=0),
        dict(name="drop_128_fp64", kind="relax", nx=128, ny=128, nz=128, h=0.4, n4=1000.0, precision="fp64",
             core="OTC", impurity=True, steps=8, refine=0),
        # An uneven box relaxed in FP32 and refined in double-float.
        dict(name="refine_96x120x160", kind="relax", nx=96, ny=120, nz=160, h=0.4, n4=800.0, precision="fp32",
             core="OTC", impurity=True, steps=30, refine=6),
        # Part of the effective-potential scan: eight positions of the impurity.
        dict(name="scan_8x128_fp32", kind="batch", grids=",".join(["128x128x128"] * 8), h=0.4, precision="fp32",
             steps=42, same=True),
        # Droplets of uneven sizes (N = 300 ... 5000) advanced together.
        dict(name="uneven_4_fp32", kind="batch", grids="96x96x96,128x128x128,160x160x160,192x192x192", h=0.4,
             precision="fp32", steps=20, same=False),
        # The large real-time run: a kicked impurity in an N = 10000 droplet.
        dict(name="kick_256x256x320_fp32", kind="kick", nx=256, ny=256, nz=320, h=0.4, n4=10000.0, precision="fp32",
             steps=30, excited=False),
        # Real time in FP64-class arithmetic on an off-power-of-two box.
        dict(name="kick_96x160x192_dfloat", kind="kick", nx=96, ny=160, nz=192, h=0.4, n4=2000.0,
             precision="dfloat", steps=12, excited=False),
        # An excited P-state impurity: anisotropic field, forces and internal
        # variables every step, in FP64.
        dict(name="excited_64x64x80_fp64", kind="kick", nx=64, ny=64, nz=80, h=0.5, n4=300.0, precision="fp64",
             steps=12, excited=True),
    ]


def _sizes(lo, hi):
    """Even 2^a 3^b 5^c in [lo, hi]."""
    def smooth(n):
        for p in (2, 3, 5):
            while n % p == 0:
                n //= p
        return n == 1
    return [n for n in range(lo + lo % 2, hi + 1, 2) if smooth(n)]


def _box(rng, lo, hi, ragged=1.6):
    """Three axes around one log-uniform size, each a different even 2,3,5 number."""
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    near = _sizes(max(lo, int(base / ragged)), min(hi, int(base * ragged)))
    return tuple(rng.choice(near) for _ in range(3))


def _atoms(dims, h):
    """A droplet whose radius is three tenths of the shortest box edge."""
    return float(round((0.3 * min(dims) * h / 2.22) ** 3) + 20)


def draw(rng):
    kind = rng.choice(["convolve", "file", "relax", "relax", "batch", "kick"])
    if kind == "convolve":
        while True:
            nx, ny, nz = _box(rng, 16, 96, 2.5)
            if (nx // 2 + 1) * ny * nz <= 33 * 64 * 64:
                return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    # a density must stay above the FP32 range out to the corners of the box
    def spacing(*dims):
        return rng.choice([h for h in (0.4, 0.4, 0.5, 0.8) if h == 0.4 or max(dims) * h <= 104])
    if kind == "file":
        nx, ny, nz = _box(rng, 32, 160)
        h = spacing(nx, ny, nz)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, h=h, n4=_atoms((nx, ny, nz), h),
                    precision=rng.choice(["fp64", "fp64", "dfloat"]), core=rng.choice(["OTC", "OTC", "OT"]),
                    periodic=rng.random() < 0.5)
    if kind == "relax":
        precision = rng.choice(["fp32", "fp32", "dfloat", "fp64"])
        nx, ny, nz = _box(rng, 32, {"fp32": 200, "dfloat": 160, "fp64": 120}[precision])
        h = spacing(nx, ny, nz)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, h=h, n4=_atoms((nx, ny, nz), h), precision=precision,
                    core=rng.choice(["OTC", "OTC", "OTC", "OT"]), impurity=rng.random() < 0.7,
                    steps={"fp32": 40, "dfloat": 16, "fp64": 8}[precision] + rng.randrange(8),
                    refine=rng.choice([0, 4]) if precision == "fp32" else 0)
    if kind == "batch":
        precision = rng.choice(["fp32", "fp32", "dfloat"])
        top, most, steps = (160, 7, 24) if precision == "fp32" else (108, 5, 16)
        boxes = [_box(rng, 48, top, 1.25) for _ in range(rng.randrange(3, most))]
        return dict(kind=kind, grids=",".join("x".join(map(str, b)) for b in boxes),
                    h=spacing(*(n for b in boxes for n in b)), precision=precision,
                    steps=rng.randrange(steps // 2, steps), same=False)
    precision = rng.choice(["fp32", "fp32", "dfloat", "fp64"])
    nx, ny, nz = _box(rng, 48, {"fp32": 240, "dfloat": 160, "fp64": 108}[precision])
    h = spacing(nx, ny, nz)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, h=h, n4=_atoms((nx, ny, nz), h), precision=precision,
                steps=rng.randrange(8, 20), excited=rng.random() < 0.3)


# ---------------------------------------------------------------------------
# Inputs.
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _axes(dims, h):
    """x, y, z broadcastable over a (nz, ny, nx) array (x fastest, the library's layout)."""
    ax = [(torch.arange(n, dtype=torch.float64, device="cuda") * h - n * h / 2) for n in dims]
    return ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _droplet(dims, h, n4, seed):
    """sqrt of a Woods-Saxon density with 0.1 % noise, normalised to n4 atoms: (nz, ny, nx) on the GPU."""
    x, y, z = _axes(dims, h)
    r = torch.sqrt(x * x + y * y + z * z)
    rho = 0.0218 / (1.0 + torch.exp(r - 2.22 * n4 ** (1.0 / 3.0)))
    psi = torch.sqrt(rho) * (1.0 + 1e-3 * torch.rand(r.shape, dtype=torch.float64, device="cuda",
                                                     generator=_generator(seed)))
    return psi * torch.sqrt(n4 / ((psi * psi).sum() * h ** 3))


def _host_psi(psi):
    """psi in page-locked memory, as the complex (nx, ny, nz) Fortran array that the library takes."""
    nz, ny, nx = psi.shape
    host = torch.empty(nz * ny * nx, 2, dtype=torch.float64, pin_memory=True)
    host.copy_(torch.view_as_real(psi.to(torch.complex128)).view(-1, 2))
    return host, host.numpy().reshape(-1).view(np.complex128).reshape((nx, ny, nz), order="F")


def _position(seed, lo, hi):
    """Where the impurity sits on the z axis."""
    return lo + (hi - lo) * np.random.default_rng(seed).random()


def _config(dims, h, n4, precision, core, periodic=True, impurity=_abi.EP_IMPURITY_FIXED, **kw):
    nx, ny, nz = dims
    return ep.make_config(nx=nx, ny=ny, nz=nz, xmax=nx * h / 2, ymax=ny * h / 2, zmax=nz * h / 2, core=core, n4=n4,
                          icon=_abi.EP_ICON_PERIODIC if periodic else _abi.EP_ICON_ZERO_OUTSIDE, impurity=impurity,
                          precision=PRECISION[precision], **kw)


def _attach(s, rimp, vimp=None, excited=False):
    pi = sigma = ep.morse(*MORSE)
    if excited:
        pi, sigma = ep.morse(*MORSE, *CORE), ep.morse(*MORSE_SIGMA, *CORE)
    s.set_impurity_potentials(pi, sigma, ep.morse(*MORSE_PLUS))
    s.set_impurity(rimp=rimp, vimp=vimp, invar=_invar(excited))


def _invar(excited):
    iv = np.zeros(10, dtype=np.complex128)
    if excited:
        iv[0], iv[3], iv[4] = 0.6, 0.64j, 0.48
    return iv


def _buffers(dims, precision):
    """Page-locked memory that psi is read into, and psi in the precision it was computed in."""
    n = dims[0] * dims[1] * dims[2]
    out64 = torch.empty(n, 2, dtype=torch.float64, pin_memory=True)
    out = torch.empty(n, 2, dtype=torch.float32) if precision == "fp32" else out64
    return dict(out64=out64, view=out64.numpy().reshape(-1).view(np.complex128).reshape(dims, order="F"), out=out)


def _instances(case, seed):
    """(dims, n4, droplet seed, impurity z or None) of each instance of a batch."""
    rng = np.random.default_rng(seed)
    shift = rng.random()
    found = []
    for i, g in enumerate(case["grids"].split(",")):
        dims = tuple(int(v) for v in g.split("x"))
        if case["same"]:
            found.append((dims, 1000.0, seed, 1.25 * i + shift))
        else:
            n4 = {96: 300.0, 128: 1000.0, 160: 2000.0, 192: 5000.0}.get(dims[0]) if len(set(dims)) == 1 else None
            n4 = n4 or _atoms(dims, case["h"])
            found.append((dims, n4, seed + 100 + i, rng.uniform(0.0, 2.22 * n4 ** (1 / 3)) if i % 2 == 0 else None))
    return found


def _kick_start(case, seed):
    """rimp, vimp of a kicked impurity."""
    return (0.0, 0.0, _position(seed, -1.0, 1.0)), (0.0, 0.0, KICK)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "convolve":
        dims = _dims(case)
        nx, ny, nz = dims
        h = 0.8
        ker = _form_factors(dims, h, _abi.EP_CORE_OTC)[1].contiguous()
        psi = _droplet(dims, h, _atoms(dims, h), seed)
        den = (psi * psi).contiguous()
        return dict(kind=kind, dims=dims, den=den, ker=ker, out=torch.empty_like(den),
                    convolve=ep.load_library()[1]["convolve_noalloc"])
    if kind == "batch":
        h, precision = case["h"], case["precision"]
        cfgs, hosts, outs, known = [], [], [], {}
        for dims, n4, s0, z in _instances(case, seed):
            cfgs.append(_config(dims, h, n4, precision, "OTC",
                                impurity=_abi.EP_IMPURITY_NONE if z is None else _abi.EP_IMPURITY_FIXED))
            if (dims, s0) not in known:
                known[dims, s0] = _host_psi(_droplet(dims, h, n4, s0))
            hosts.append(known[dims, s0])
            outs.append(_buffers(dims, precision))
        b = ep.Batch(cfgs)
        for s, (_, _, _, z) in zip(b, _instances(case, seed)):
            if z is not None:
                _attach(s, (0.0, 0.0, z))
        return dict(kind=kind, batch=b, hosts=hosts, outs=outs, precision=precision, steps=case["steps"])
    dims = _dims(case)
    host, psi = _host_psi(_droplet(dims, case["h"], case["n4"], seed))
    state = dict(kind=kind, host=host, psi=psi, precision=case["precision"])
    if kind == "file":
        s = ep.Solver(_config(dims, case["h"], case["n4"], case["precision"], case["core"], case["periodic"]))
        _attach(s, (0.0, 0.0, _position(seed, -2.0, 2.0)))
        return dict(state, solver=s)
    state.update(_buffers(dims, case["precision"]), steps=case["steps"])
    if kind == "relax":
        s = ep.Solver(_config(dims, case["h"], case["n4"], case["precision"], case["core"],
                              impurity=_abi.EP_IMPURITY_FIXED if case["impurity"] else _abi.EP_IMPURITY_NONE))
        if case["impurity"]:
            _attach(s, (0.0, 0.0, _position(seed, 0.0, 4.0)))
        return dict(state, solver=s, refine=case["refine"])
    s = ep.Solver(_config(dims, case["h"], case["n4"], case["precision"], "OTC", impurity=_abi.EP_IMPURITY_MOVING,
                          time_mode=_abi.EP_REAL_TIME, renormalize=0, mimpur=MIMPUR,
                          fix_lambda=0 if case["excited"] else 1, als_p=50.0 if case["excited"] else 0.0))
    rimp, vimp = _kick_start(case, seed)
    _attach(s, rimp, vimp, excited=case["excited"])
    return dict(state, solver=s, at=dict(rimp=rimp, vimp=vimp, invar=_invar(case["excited"])))


# ---------------------------------------------------------------------------
# One pass.
def _energies(s, precision):
    """Energies as an array in the arithmetic of the fields they come from."""
    e = s.energy()
    return np.array([e[k] for k in ENERGIES], dtype=np.float32 if precision == "fp32" else np.float64)


def _read_psi(s, buf):
    s.psi(out=buf["view"])
    if buf["out"] is not buf["out64"]:
        buf["out"].copy_(buf["out64"])
    return buf["out"]


def run(state):
    kind = state["kind"]
    if kind == "convolve":
        nx, ny, nz = state["dims"]
        st = state["convolve"](state["den"].data_ptr(), state["ker"].data_ptr(), state["out"].data_ptr(), nx, ny, nz,
                               torch.cuda.current_stream().cuda_stream)
        if st != _abi.EP_OK:
            raise RuntimeError("ep_convolve_noalloc: status %d" % st)
        return state["out"]
    precision = state["precision"]
    if kind == "batch":
        b = state["batch"]
        for s, (_, psi) in zip(b, state["hosts"]):
            s.start(psi)
        for _ in range(RK_STEPS):
            b.steprk(DT)
        stats = b.run(state["steps"], DT)
        for s in b:
            s.poten()
        return {"energy": np.array([_energies(s, precision) for s in b]),
                "mu": np.array([q["mu"] for q in stats], dtype=np.float32 if precision == "fp32" else np.float64),
                "psi": [_read_psi(s, o) for s, o in zip(b, state["outs"])]}
    s = state["solver"]
    if kind == "file":
        s.start(state["psi"])
        return {"energy": _energies(s, precision)}
    if kind == "relax":
        refine = state["refine"]
        s.start(state["psi"])
        for _ in range(RK_STEPS):
            s.steprk(DT)
        s.run(state["steps"], DT)
        if refine:
            s.set_precision("dfloat")
            s.run(refine, DT)
        s.poten()
        # a job's result carries the precision of its bulk steps
        out = {"energy": _energies(s, precision), "psi": _read_psi(s, state)}
        if refine:
            s.set_precision(precision)
        return out
    s.set_impurity(**state["at"])
    s.start(state["psi"])
    for _ in range(RK_STEPS + 1):
        s.steprk(DT_REAL)
    s.run(state["steps"], DT_REAL)
    s.poten()
    out = {"energy": _energies(s, precision), "psi": _read_psi(s, state)}
    imp = s.impurity()
    out["impurity"] = np.concatenate([imp["rimp"], imp["vimp"]]).astype(np.float32 if precision == "fp32" else float)
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without.
def _step_work(dims, real, impurity=True):
    """One predictor-corrector step: the multistep state (psi, psiold, hpsiold and pc as the two
    halves of the method need them), the density and the mean field once each, and the arithmetic of
    14 real FFTs, two complex 13-point Laplacians, six first derivatives and the point-wise algebra."""
    nx, ny, nz = dims
    n = nx * ny * nz
    c = 2 * real
    b = ((5 + 3) * c + (6 + 2) * c + (2 + 2) * real + (2 * real if impurity else 0)) * n
    f = (14 * 2.5 * math.log2(n) + 2 * 156 + 6 * 18 + 100) * n
    return b, f


def _poten_work(dims, real):
    """One mean field: the density in, the potential out."""
    n = dims[0] * dims[1] * dims[2]
    return 2 * real * n, (14 * 2.5 * math.log2(n) + 6 * 18 + 100) * n


def _job_work(dims, precision, steps, refine=0):
    real = 4 if precision == "fp32" else 8
    n = dims[0] * dims[1] * dims[2]
    sb, sf = _step_work(dims, real)
    db, df = _step_work(dims, 8)
    pb, pf = _poten_work(dims, real)
    rk = 4 * RK_STEPS
    # the density in and psi out (16 bytes a point), start-up, RK stages (psi, q and the fields), steps, energies
    return (32 * n + rk * (10 * real * n + pb) + steps * sb + refine * db + 2 * pb + 12 * real * n,
            (rk + 2) * pf + rk * 170 * n + steps * sf + refine * df + 150 * n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        got = [_job_work(tuple(int(v) for v in g.split("x")), case["precision"], case["steps"])
               for g in case["grids"].split(",")]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    if kind == "convolve":
        nh = (dims[0] // 2 + 1) * dims[1] * dims[2]
        return {"bytes": 16 * n + 8 * nh, "flops": 2 * 2.5 * n * math.log2(n) + 2 * nh}
    real = 4 if case["precision"] == "fp32" else 8
    pb, pf = _poten_work(dims, real)
    if kind == "file":
        return {"bytes": 16 * n + 3 * real * n + pb + 12 * real * n, "flops": pf + 200 * n}
    if kind == "relax":
        b, f = _job_work(dims, case["precision"], case["steps"], case["refine"])
        return {"bytes": b, "flops": f}
    # the job's work, and in each step and RK stage the impurity's field written and its force and moments summed
    b, f = _job_work(dims, case["precision"], case["steps"])
    moved = case["steps"] + 3 * (RK_STEPS + 1)
    return {"bytes": b + moved * 10 * real * n, "flops": f + moved * 80 * n}


# ---------------------------------------------------------------------------
# The same physics in plain torch, in 64 bits.  Arrays are (nz, ny, nx).
def _si(x):
    """The sine integral of x > 0: its power series up to 4, beyond it the continued fraction of E1(ix)
    (pi/2 + Im E1), evaluated from its 160th convergent."""
    small = torch.minimum(x, torch.full_like(x, 4.0))
    term, s = small.clone(), small.clone()
    for k in range(1, 30):
        term = term * (-small * small / ((2 * k) * (2 * k + 1)))
        s = s + term / (2 * k + 1)
    z = 1j * torch.maximum(x, torch.full_like(x, 4.0)).to(torch.complex128)
    f = z + 2 * 160 + 1
    for k in range(160, 0, -1):
        f = z + 2 * k - 1 - k * k / f
    e1 = torch.exp(-z) / f
    return torch.where(x <= 4.0, s, math.pi / 2 + e1.imag)


def _form_factors(dims, h, core, c=None):
    """fvlj4, wcgk, kalfs on the (nz, ny, nx/2+1) half spectrum."""
    c = c or ep.make_config()
    nx, ny, nz = dims
    fz, fy = (torch.fft.fftfreq(n, h, dtype=torch.float64, device="cuda") for n in (nz, ny))
    fx = torch.fft.rfftfreq(nx, h, dtype=torch.float64, device="cuda")
    p = torch.sqrt(fx.view(1, 1, -1) ** 2 + fy.view(1, -1, 1) ** 2 + fz.view(-1, 1, 1) ** 2)
    h4 = c.h4op if core == _abi.EP_CORE_OP else c.h4ot
    eps, s6 = c.eps4, c.sigma4 ** 6
    zero = p < 1e-10
    a = 2 * math.pi * torch.where(zero, torch.ones_like(p), p)
    y = a * h4
    si, sn, cs, y2 = math.pi / 2 - _si(y), torch.sin(y), torch.cos(y), y * y
    bd = 40320.0 - 720.0 * y2 + 24.0 * y2 ** 2 - 2.0 * y2 ** 3 + y2 ** 4
    cd = 362880.0 - 5040.0 * y2 + 120.0 * y2 ** 2 - 6.0 * y2 ** 3 + y2 ** 4
    t11 = (a * bd * cs + cd * sn / h4) / (3628800.0 * h4 ** 9) - a ** 10 * si / 3628800.0
    t5 = -(a * (y2 - 2.0) * cs + (y2 - 6.0) * sn / h4) / (24.0 * h4 ** 3) + a ** 4 * si / 24.0
    fv = 8.0 * eps * s6 * (s6 * t11 - t5) / (a / (2 * math.pi))
    at0 = 16 * math.pi * eps * (s6 * s6 / (9.0 * h4 ** 9) - s6 / (3.0 * h4 ** 3))
    fv = torch.where(zero, torch.full_like(fv, at0), fv)
    aux = sn - y * cs
    wc = torch.where(zero | (aux.abs() < 1e-10), torch.ones_like(p), 3.0 * aux / y ** 3)
    return fv, wc, torch.exp(-(math.pi * c.l * p) ** 2)


def _weights():
    """Central weights of the 13-point first and second derivatives at +k."""
    w1, w2 = [0.0], [0.0]
    for k in range(1, 7):
        m = (-1) ** (k + 1) * math.factorial(6) ** 2 / (math.factorial(6 - k) * math.factorial(6 + k))
        w1.append(m / k)
        w2.append(2.0 * m / k ** 2)
        w2[0] -= 2.0 / k ** 2
    return w1, w2


class _Exact:
    """One droplet: the mean field, the energies and the two integrators."""

    def __init__(self, cfg, rimp=(0.0, 0.0, 0.0), vimp=(0.0, 0.0, 0.0), invar=None, excited=False):
        self.c = cfg
        self.dims = (cfg.nx, cfg.ny, cfg.nz)
        self.h = 2.0 * cfg.xmax / cfg.nx
        self.dv = self.h ** 3
        self.periodic = cfg.icon == _abi.EP_ICON_PERIODIC
        self.otc = cfg.core == _abi.EP_CORE_OTC
        self.real_time = cfg.time_mode == _abi.EP_REAL_TIME
        self.ff = _form_factors(self.dims, self.h, cfg.core, cfg)
        self.w1, self.w2 = _weights()
        self.rimp, self.vimp = np.array(rimp, float), np.array(vimp, float)
        self.aimp = np.zeros(3)
        self.iv = np.zeros(10, complex) if invar is None else invar.copy()
        self.hiv = np.zeros(10, complex)
        self.excited = excited
        n = max(self.dims)
        self.npot = 100 * n + 1
        self.delr = 4.0 * max(cfg.xmax, cfg.ymax, cfg.zmax) / (self.npot - 1)
        self.uimp = torch.zeros(self.dims[::-1], dtype=torch.float64, device="cuda")
        self.po, self.ph, self.pc = [None] * 3, [None] * 2, 0.0
        self.q = 0.0
        self.moving = cfg.impurity == _abi.EP_IMPURITY_MOVING

    def shift(self, f, axis, k):
        """f(i + k) along x, y, z = axis 0, 1, 2."""
        d = 2 - axis
        g = torch.roll(f, -k, d)
        if not self.periodic:
            g.narrow(d, f.shape[d] - k if k > 0 else 0, abs(k)).zero_()
        return g

    def d1(self, f, axis):
        return sum(self.w1[k] * (self.shift(f, axis, k) - self.shift(f, axis, -k)) for k in range(1, 7)) / self.h

    def lap(self, f):
        s = 3 * self.w2[0] * f
        for axis in range(3):
            for k in range(1, 7):
                s += self.w2[k] * (self.shift(f, axis, k) + self.shift(f, axis, -k))
        return s / self.h ** 2

    def conv(self, f, w):
        return torch.fft.irfftn(torch.fft.rfftn(f) * w, s=f.shape)

    def poten(self):
        c, d = self.c, self.den
        fv, wc, ka = self.ff
        F = torch.fft.rfftn(d)
        cg, self.lj = (torch.fft.irfftn(F * w, s=d.shape) for w in (wc, fv))
        pot = self.lj + cg * cg * (c.cp4 / 2 + c.cpp4 / 3 * cg) + self.conv(d * cg * (c.cp4 + c.cpp4 * cg), wc)
        self.cg = cg
        if self.otc or self.moving:
            self.grad = [self.d1(d, a) for a in range(3)]
        if self.otc:
            f = 1.0 - torch.fft.irfftn(F * ka, s=d.shape) / c.den0s
            I = [self.conv(f * g, ka) for g in self.grad]
            u = self.conv(sum(g * i for g, i in zip(self.grad, I)), ka) / c.den0s
            div = sum(self.d1(f * i, a) for a, i in enumerate(I))
            pot = pot + (u + div) * c.h2o2m4 * c.alphas
            self.f, self.I = f, I
        e2 = torch.exp(2.0 * c.beta * (d - c.den_m))
        self.onept = 2.0 * e2 / (1.0 + e2)                           # 1 + tanh
        self.pot = pot + c.C * (self.onept + c.beta * d * self.onept * (2.0 - self.onept))

    def _table(self, f, r):
        """Three-point interpolation in the table f(i) at r = (i - 1) delr."""
        i0 = (1.5 + r / self.delr).to(torch.int64).clamp(1, self.npot)
        d = r / self.delr - (i0 - 1)
        return f[i0] + d * (0.5 * (f[i0 + 1] - f[i0 - 1]) + 0.5 * d * (f[i0 + 1] - 2 * f[i0] + f[i0 - 1]))

    def potenimp(self):
        r = torch.arange(self.npot, dtype=torch.float64, device="cuda") * self.delr
        pi = sg = _morse(r, MORSE)
        if self.excited:
            pi, sg = (torch.where(r < CORE[0], torch.full_like(r, CORE[1]), _morse(r, q)) for q in (MORSE, MORSE_SIGMA))
        tp, td = (torch.cat([t[:1], t, t[-1:]]) for t in (pi, sg - pi))
        self.xyz = [a - s for a, s in zip(_axes(self.dims, self.h), self.rimp)]
        x, y, z = self.xyz
        r2 = x * x + (y * y + z * z)
        rr = torch.sqrt(r2)
        self.vpi = self._table(tp, rr)
        # at r = 0 the library takes the potential's umax (1000 K)
        self.delta = torch.where(rr > 1e-3, self._table(td, rr) / r2.clamp_min(1e-12), torch.full_like(rr, 1000.0))
        u = self.vpi
        for s in (0, 1):
            v = sum(complex(self.iv[s + 2 * k]) * q for k, q in enumerate(self.xyz))
            u = u + self.delta * (v.real ** 2 + v.imag ** 2)
        self.uimp = u.clamp_max(1000.0)

    def forces(self):
        """aimp and, for internal variables that evolve, -i H iv."""
        self.aimp = np.array([-float((g * self.uimp).sum()) * self.dv for g in self.grad]) / (MIMPUR * ep.MP_U)
        if self.c.fix_lambda:
            return
        m = np.zeros((3, 3))
        for a in range(3):
            for b in range(3):
                t = self.delta * self.xyz[a] * self.xyz[b] + (self.vpi if a == b else 0.0)
                m[a, b] = float((self.den * t).sum()) * self.dv
        iv, A = self.iv[:6], self.c.als_p / 2.0
        H = np.empty(6, complex)
        H[0::2], H[1::2] = m @ iv[0::2], m @ iv[1::2]
        H += A * np.array([-1j * iv[2] + iv[5], 1j * iv[3] - iv[4], 1j * iv[0] - 1j * iv[5],
                           -1j * iv[1] - 1j * iv[4], -iv[1] + 1j * iv[3], iv[0] + 1j * iv[2]])
        self.hiv[:6] = -1j * (H - self.c.ev0 * iv)

    def start(self, psi):
        self.psi = psi.to(torch.complex128)
        self.den = psi * psi
        if self.c.impurity != _abi.EP_IMPURITY_NONE:
            self.potenimp()
        self.poten()

    def refresh(self):
        if self.moving:
            self.potenimp()
        self.poten()
        if self.moving:
            self.forces()

    def H(self):
        L = self.lap(self.psi) * self.c.h2o2m4 - (self.pot + self.uimp) * self.psi
        return 1j * L if self.real_time else L

    def set_psi(self, psi):
        self.psi = psi
        self.den = psi.real ** 2 + psi.imag ** 2

    def steprk(self, dt):
        s2 = math.sqrt(2.0)
        stages = zip((0.5, 1 - 1 / s2, 1 + 1 / s2, 1 / 6), (2.0, 1.0, 1.0, 2.0), (0.5, 1 - 1 / s2, 1 + 1 / s2, 0.5))
        if not hasattr(self, "qs"):
            self.qs = [np.zeros(3), np.zeros(3), np.zeros(10, complex)]
            self.small = [[None] * 3 for _ in range(3)]              # rimp, vimp, invar, newest first
            self.slopes = [[None] * 2 for _ in range(2)]             # aimp, -i H iv, newest first
            self.pcs = [np.zeros(3), np.zeros(3), np.zeros(10, complex)]
        for jr, (a, b, cr) in enumerate(stages):
            H = self.H()
            x = a * (H - b * self.q)
            self.q = self.q + 3 * x - cr * H
            if jr == 0:
                self.po, self.ph = [self.psi] + self.po[:2], [H, self.ph[0]]
            self.set_psi(self.psi + dt * x)
            if self.moving:
                now, slope = [self.rimp, self.vimp, self.iv], [self.vimp, self.aimp, self.hiv.copy()]
                for k in range(2 if self.c.fix_lambda else 3):
                    x = a * (slope[k] - b * self.qs[k])
                    self.qs[k] = self.qs[k] + 3 * x - cr * slope[k]
                    if jr == 0:
                        self.small[k] = [now[k]] + self.small[k][:2]
                        if k:
                            self.slopes[k - 1] = [slope[k], self.slopes[k - 1][0]]
                    now[k] = now[k] + dt * x
                self.rimp, self.vimp, self.iv = now
            if jr < 3:
                self.refresh()

    def steppc(self, dt):
        c112, c9, c43 = 112 / 121, 9 / 121, 4 / 3
        H = self.H()
        pp = self.po[2] + c43 * dt * (2 * H - self.ph[0] + 2 * self.ph[1])
        new = pp - c112 * self.pc
        old, self.pc, self.ph = self.psi, pp, [H, self.ph[0]]
        if self.moving:
            r, v, w = self.small
            lam = not self.c.fix_lambda
            v_old, a_old = self.vimp, self.aimp
            ax = r[2] + c43 * dt * (2 * v_old - v[0] + 2 * v[1])
            r_old, self.rimp, self.pcs[0] = self.rimp, ax - c112 * self.pcs[0], ax
            ax = v[2] + c43 * dt * (2 * a_old - self.slopes[0][0] + 2 * self.slopes[0][1])
            v_new, self.pcs[1] = ax - c112 * self.pcs[1], ax
            self.slopes[0] = [a_old, self.slopes[0][0]]
            if lam:
                ax = w[2] + c43 * dt * (2 * self.hiv - self.slopes[1][0] + 2 * self.slopes[1][1])
                iv_old, self.iv, self.pcs[2] = self.iv, ax - c112 * self.pcs[2], ax
                self.slopes[1] = [self.hiv.copy(), self.slopes[1][0]]
        self.set_psi(new)
        self.refresh()
        H = self.H()
        p5 = (9 * old - self.po[1] + 3 * dt * (H + 2 * self.ph[0] - self.ph[1])) / 8
        self.pc = self.pc - p5
        self.po = [old] + self.po[:2]
        self.set_psi(p5 + c9 * self.pc)
        if self.moving:
            ax = (9 * r_old - r[1] + 3 * dt * (v_new + 2 * v_old - v[0])) / 8
            self.pcs[0] = self.pcs[0] - ax
            self.rimp = ax + c9 * self.pcs[0]
            ax = (9 * v_old - v[1] + 3 * dt * (self.aimp + 2 * self.slopes[0][0] - self.slopes[0][1])) / 8
            self.pcs[1] = self.pcs[1] - ax
            self.vimp = ax + c9 * self.pcs[1]
            self.small[0], self.small[1] = [r_old] + r[:2], [v_old] + v[:2]
            if lam:
                ax = (9 * iv_old - w[1] + 3 * dt * (self.hiv + 2 * self.slopes[1][0] - self.slopes[1][1])) / 8
                self.pcs[2] = self.pcs[2] - ax
                self.iv = ax + c9 * self.pcs[2]
                self.small[2] = [iv_old] + w[:2]
        if not self.real_time and self.c.renormalize:
            s = math.sqrt(self.c.n4 / (float(self.den.sum()) * self.dv))
            self.po, self.ph, self.pc = [s * p for p in self.po], [s * p for p in self.ph], s * self.pc
            self.set_psi(s * self.psi)

    def energy(self):
        c, d, dv = self.c, self.den, self.dv
        e = dict.fromkeys(ENERGIES, 0.0)
        e["ekin4"] = c.h2o2m4 * sum(float(self.d1(self.psi, a).abs().square().sum()) for a in range(3)) * dv
        e["elj4"] = 0.5 * float((self.lj * d).sum()) * dv
        e["ecor4"] = float((d * self.cg ** 2 * (0.5 * c.cp4 + c.cpp4 / 3 * self.cg)).sum()) * dv
        if self.otc:
            e["ealphas"] = -0.5 * c.h2o2m4 * c.alphas * dv * float(
                (self.f * sum(g * i for g, i in zip(self.grad, self.I))).sum())
        e["esolid"] = c.C * float((d * self.onept).sum()) * dv
        e["etot4"] = e["ekin4"] + e["elj4"] + e["ecor4"] + e["ealphas"]
        e["ekinx"] = 0.5 * c.mimpur * ep.MP_U * float(self.vimp @ self.vimp)
        if c.impurity != _abi.EP_IMPURITY_NONE:
            r = torch.sqrt(sum((a - s) ** 2 for a, s in zip(_axes(self.dims, self.h), self.rimp)))
            e["eHeX"] = float((d * self.uimp).sum()) * dv
            e["uplus"] = float((d * _morse(r, MORSE_PLUS)).sum()) * dv
        iv, cj = self.iv, self.iv.conj()
        e["eso"] = c.als_p * ((cj[0] * iv[5] - cj[1] * iv[4]).real +
                              (cj[0] * iv[2] + cj[3] * iv[1] + cj[2] * iv[5] + cj[3] * iv[4]).imag)
        e["eimpu"] = e["ekinx"] + e["eHeX"] + e["eso"]
        e["etot"] = e["etot4"] + e["eimpu"]
        e["n4"] = float(d.sum()) * dv
        return np.array([e[k] for k in ENERGIES])

    def psi_out(self):
        return torch.view_as_real(self.psi).reshape(-1, 2)


def _morse(r, par):
    e = torch.exp(-par[2] * (r - par[1]))
    return par[0] * (e * e - 2.0 * e)


def _exact_job(dims, h, n4, core, seed, z, steps):
    x = _Exact(_config(dims, h, n4, "fp64", core, impurity=_abi.EP_IMPURITY_NONE if z is None
                       else _abi.EP_IMPURITY_FIXED), rimp=(0.0, 0.0, z or 0.0))
    x.start(_droplet(dims, h, n4, seed))
    for _ in range(RK_STEPS):
        x.steprk(DT)
    for _ in range(steps):
        x.steppc(DT)
    x.poten()
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        found = [_exact_job(dims, case["h"], n4, "OTC", s0, z, case["steps"])
                 for dims, n4, s0, z in _instances(case, seed)]
        return {"energy": np.array([x.energy() for x in found]), "mu": None, "psi": [x.psi_out() for x in found]}
    dims = _dims(case)
    if kind == "convolve":
        psi = _droplet(dims, 0.8, _atoms(dims, 0.8), seed)
        F = torch.fft.rfftn(psi * psi)
        return torch.fft.irfftn(F * _form_factors(dims, 0.8, _abi.EP_CORE_OTC)[1], s=psi.shape)
    if kind == "file":
        x = _Exact(_config(dims, case["h"], case["n4"], "fp64", case["core"], case["periodic"]),
                   rimp=(0.0, 0.0, _position(seed, -2.0, 2.0)))
        x.start(_droplet(dims, case["h"], case["n4"], seed))
        return {"energy": x.energy()}
    if kind == "relax":
        x = _exact_job(dims, case["h"], case["n4"], case["core"], seed,
                       _position(seed, 0.0, 4.0) if case["impurity"] else None, case["steps"] + case["refine"])
        return {"energy": x.energy(), "psi": x.psi_out()}
    cfg = _config(dims, case["h"], case["n4"], "fp64", "OTC", impurity=_abi.EP_IMPURITY_MOVING,
                  time_mode=_abi.EP_REAL_TIME, renormalize=0, mimpur=MIMPUR, fix_lambda=0 if case["excited"] else 1,
                  als_p=50.0 if case["excited"] else 0.0)
    x = _Exact(cfg, *_kick_start(case, seed), invar=_invar(case["excited"]), excited=case["excited"])
    x.start(_droplet(dims, case["h"], case["n4"], seed))
    for _ in range(RK_STEPS + 1):
        x.steprk(DT_REAL)
    for _ in range(case["steps"]):
        x.steppc(DT_REAL)
    x.poten()
    return {"energy": x.energy(), "psi": x.psi_out(), "impurity": np.concatenate([x.rimp, x.vimp])}
