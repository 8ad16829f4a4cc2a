"""What a user of this framework has it compute, as measurable cases.

Every case goes through the public entry points: ``stx.solver.Solver`` (steps,
captured steps, the RK right-hand side), ``stx.reactors.BatchReactors`` and, for
the flux kernels that a Fortran host calls one by one, the C ABI of
``include/stx.h`` as ``stx.native`` loads it.  The kinds:

  turb     one iteration of the integration loop of the reacting turbulence box
  flame    a captured graph of 10 fixed-dt steps of a 1-D premixed flame
  tube     a captured graph of CFL-driven steps of the reactive shock tube (1-D, or a 2-D strip)
  cell     one iteration of the loop of the 0-D reactor example (a 1 x 1 x 1 box)
  reactors one batch of constant-pressure 0-D reactors
  aux      primitive and transport recovery on a box, ghosts included
  flux     convective and viscous flux divergences on a box
  rk53     one transport-only RK3 step of the 53-species mechanism

``exact`` restates the recovery and the fluxes in plain torch FP64.  Steps with
chemistry have no such value: the adaptive ROK4 integration defines them.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "prop-streams2_b200"))

from stx import case as CS  # noqa: E402
from stx import configs  # noqa: E402
from stx import mech as M  # noqa: E402
from stx.native import check  # noqa: E402
from stx.reactors import BatchReactors, sample_h2air  # noqa: E402
from stx.solver import Solver  # noqa: E402

F64 = torch.float64
DEV = "cuda"


def listed():
    return [
        # the headline workload at its size: 256^3 reacting turbulence, FP64
        dict(name="turb_256", kind="turb", n=256, form="fp64"),
        # an odd box (no even ghosted row, so no tensor-copy staging), the size of a resolution study
        dict(name="turb_61", kind="turb", n=61, form="fp64"),
        # the mixed precision form at an ordinary production size
        dict(name="turb_128_mixed", kind="turb", n=128, form="mixed"),
        # the laminar premixed flame at the published example's size and mechanism (2000 cells, 11 species)
        dict(name="flame_2000", kind="flame", nx=2000, mech="flame_11sp"),
        # the 1-D reactive shock tube, 2400 cells, dt recomputed every step
        dict(name="tube_2400", kind="tube", nx=2400, ny=1, steps=10),
        # the served 2-D strip of the shock tube
        dict(name="tube_512x128", kind="tube", nx=512, ny=128, steps=5),
        # the 0-D reactor example: one cell through the whole loop, so launches are all there is
        dict(name="cell_14sp", kind="cell", version=2),
        # a throughput batch of reactors, over a window that all of them finish
        dict(name="reactors_8192", kind="reactors", n=8192, t_max=1e-7, form="fp64"),
        # a served batch of reactors
        dict(name="reactors_200", kind="reactors", n=200, t_max=1e-6, form="fp64"),
        # the state recovery alone, on a box with unequal extents
        dict(name="aux_200x96x72", kind="aux", nx=200, ny=96, nz=72),
        # the flux kernels alone, on a box that is no multiple of any tile
        dict(name="flux_150x101x77", kind="flux", nx=150, ny=101, nz=77),
        # the large mechanism's transport half (53 species)
        dict(name="rk53_40", kind="rk53", n=40),
    ]


def draw(rng):
    def size(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b + 0.49)))))

    kind = rng.choice(["turb", "turb", "flame", "tube", "cell", "reactors", "aux", "flux", "rk53"])
    if kind == "turb":
        return dict(kind=kind, n=size(32, 200), form=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "flame":
        return dict(kind=kind, nx=size(512, 2200), mech=rng.choice(["flame_11sp", "h2air_9sp"]))
    if kind == "tube":
        ny = rng.choice([1, size(5, 160)])
        return dict(kind=kind, nx=size(400, 4800 if ny == 1 else 700), ny=ny, steps=rng.choice([5, 10]))
    if kind == "cell":
        return dict(kind=kind, version=rng.choice([1, 2]), nx=size(1, 40), ny=rng.choice([1, 2, 3]))
    if kind == "reactors":
        return dict(kind=kind, n=size(1, 10000), t_max=rng.choice([3e-8, 1e-7, 2e-7]),
                    form=rng.choice(["fp64", "fp64", "split"]))
    if kind == "rk53":
        return dict(kind=kind, n=size(8, 48))
    a = [size(20, 180) for _ in range(3)]
    while a[0] * a[1] * a[2] > 1500000:
        a[a.index(max(a))] //= 2
    return dict(kind=kind, nx=a[0], ny=a[1], nz=a[2])


# ---------------------------------------------------------------- inputs
_TABLES = {}


def _tables(mech, p0, tmax):
    """Property tables, which a program builds once per mechanism."""
    key = (mech, p0, tmax)
    if key not in _TABLES:
        if mech == "stiff53":
            _TABLES[key] = configs.stiff_mechanism_tables(0)[1]
        else:
            _TABLES[key] = M.build_tables(configs.mechanism(mech), p0, 200.0, tmax, 1.0)
    return _TABLES[key]


def _advanced(sol, steps):
    """A running solver: prepared, `steps` iterations in."""
    sol.prepare()
    for _ in range(steps):
        sol.step()
    return sol


def _turb(case, seed):
    """The turbulence workload some way into its decay: its velocity field, with temperature
    and pressure fluctuations (the fresh field's uniform state is met once per run).  A
    smaller box is a same-resolution sample, so it holds fewer large eddies."""
    n = case["n"]
    c = configs.turbulence_case(n, tables=_tables("h2air_9sp", 101325.0, 5500.0), k0=max(1.0, min(4.0, n / 32.0)))
    w, wa = configs.turbulence_fields(c, seed, xp=torch, device=DEV)
    rng = np.random.default_rng(seed)
    rho = c.interior(w)[:9].sum(0)
    c.interior(w)[12] += rho * (1.2e3 * 30.0 * _modes((n, n, n), rng, 4))
    c.interior(w).mul_(1.0 + 0.03 * _modes((n, n, n), rng, 4))
    del rho
    sol = Solver(c, w=w, w_aux=wa)
    sol.set_precision(case["form"])
    return _advanced(sol, 2)


def _flame(case, seed):
    rng = np.random.default_rng(seed)
    tb = _tables(case["mech"], 101325.0, 5500.0)
    c = configs.flame_case(case["nx"], phi=rng.uniform(0.5, 1.5), Tu=rng.uniform(300.0, 800.0), tables=tb,
                           mech_name=case["mech"])
    sol = _advanced(Solver(c), 5)
    return sol, sol.capture(10)


def _tube(case, seed):
    rng = np.random.default_rng(seed)
    tb = _tables("shock_tube_9sp", 7173.0, 20000.0)
    c = configs.tube_case(case["nx"], case["ny"], tables=tb)
    c.cfl = 0.5
    s = rng.uniform(0.95, 1.05, 3)
    c._init_reactive_tube(0.18075 * s[0], -487.34 * s[1], 35594.0 * s[2])
    sol = _advanced(Solver(c), 5)
    return sol, sol.capture(case["steps"])


# examples/batch_reactor: H2/CO/O2/N2, Strang + ROK4, fixed dt 2e-7 s on one periodic cell
CELL_Y = {2: 0.01495, 4: 0.1149, 6: 0.00375, 7: 0.58285, 10: 0.00635, 11: 0.27715}


def _cell(case, seed):
    rng = np.random.default_rng(seed)
    Y = np.zeros(14)
    for k, v in CELL_Y.items():
        Y[k - 1] = v
    nx, ny = case.get("nx", 1), case.get("ny", 1)
    cfg = CS.default_ini(nx, ny, 1, L=(0.05, 0.05, 0.05), t0=rng.uniform(1000.0, 1300.0), Y=Y, ns=14, nkeep=0,
                         sensor_threshold=-0.2, sensor_type=0, cfl=-2e-7, flow_init=8,
                         rosenbrock_version=case["version"])
    return _advanced(Solver(CS.Case(cfg, _tables("keromnes_14sp", 101325.0, 5500.0))), 5)


def _modes(shape, rng, kmax):
    """A smooth periodic field in [-1, 1] of a few seeded modes, (nz, ny, nx)."""
    x = [torch.arange(n, device=DEV, dtype=F64) / n * 2.0 * math.pi for n in shape]
    f = torch.zeros(shape, device=DEV, dtype=F64)
    for _ in range(4):
        k = rng.integers(1, kmax + 1, size=3)
        ph = rng.uniform(0, 2 * math.pi, size=3)
        f += rng.uniform(0.3, 1.0) * (torch.sin(k[0] * x[0] + ph[0])[:, None, None] *
                                      torch.sin(k[1] * x[1] + ph[1])[None, :, None] *
                                      torch.sin(k[2] * x[2] + ph[2])[None, None, :])
    return f / f.abs().max()


def _box(case, seed):
    """A periodic box of partly burnt H2/air at the turbulence case's resolution:
    800 to 2000 K, all nine species present, velocities that trip the sensor on part
    of the faces."""
    rng = np.random.default_rng(seed)
    mech = configs.mechanism("h2air_9sp")
    tb = _tables("h2air_9sp", 101325.0, 5500.0)
    n = (case["nz"], case["ny"], case["nx"])
    Yu = configs.h2air_Y(0.7, mech)
    d = 2.0 * math.pi * 1e-3 / 256.0
    cfg = CS.default_ini(n[2], n[1], n[0], L=(d * n[2], d * n[1], d * n[0]), t0=1000.0, Y=Yu, ns=9, nkeep=2, cfl=0.5)
    c = CS.Case(cfg, tb, alloc_fields=False)
    T = 1400.0 + 600.0 * _modes(n, rng, 3)
    vel = [300.0 * _modes(n, rng, 4) for _ in range(3)]
    prog = 0.5 + 0.4 * _modes(n, rng, 3)
    Y = torch.empty((9,) + n, device=DEV, dtype=F64)
    for k in range(9):
        Y[k] = Yu[k] * (1.0 - 0.6 * prog) if Yu[k] > 0 else 0.01 * prog * (1.0 + 0.5 * _modes(n, rng, 3))
    Y /= Y.sum(0)
    rho = 101325.0 * (1.0 + 0.1 * _modes(n, rng, 3)) / (torch.einsum("k,kzyx->zyx", _t(tb.rgas), Y) * T)
    w = torch.zeros((13, c.nzg, c.nyg, c.nxg), device=DEV, dtype=F64)
    wa = torch.zeros((c.nv_aux, c.nzg, c.nyg, c.nxg), device=DEV, dtype=F64)
    w[:] = _t(c.winf)[:, None, None, None]
    wa[9 + 4] = 1000.0
    c.interior(w)[:9] = rho * Y
    for m in range(3):
        c.interior(w)[9 + m] = rho * vel[m]
    c.interior(w)[12] = rho * (_energy(tb, T, Y) + 0.5 * sum(v * v for v in vel))
    c.interior(wa)[9 + 4] = T
    sol = Solver(c, w=w, w_aux=wa)
    sol.prepare()
    return sol


def _rk53(case, seed):
    c = configs.stiff_case(case["n"], seed=seed % 1000, tables=_tables("stiff53", 101325.0, 5500.0), dt=1e-9)
    sol = Solver(c)
    sol.prepare()
    return sol


def _reactors(case, seed):
    br = BatchReactors("h2air_9sp", tables=_tables("h2air_9sp", 101325.0, 5500.0))
    br.set_form(case["form"])
    T0, p0, Y0 = sample_h2air(case["n"], seed, br.mech)
    return br, _t(T0), _t(p0), _t(Y0)


def prepare(case, seed):
    kind = case["kind"]
    make = {"turb": _turb, "flame": _flame, "tube": _tube, "cell": _cell, "aux": _box, "flux": _box, "rk53": _rk53,
            "reactors": _reactors}[kind]
    return case, make(case, seed)


# ---------------------------------------------------------------- one pass
def _fields(sol):
    """The state after a pass: the species densities one by one, the momentum, the energy, T and p."""
    c = sol.case
    ns = c.ns
    if ns > 20:                        # by groups
        g = [sol.w[:ns], sol.w[ns:ns + 3], sol.w[ns + 3]]
    elif c.flow_init == 8:             # gas at rest: its momenta, which are rounding, beside its energy
        g = [sol.w[m] for m in range(ns)] + [sol.w[ns:]]
    else:
        g = [sol.w[m] for m in range(ns)] + [sol.w[ns:ns + 3], sol.w[ns + 3]]
    return [c.interior(x) for x in g] + [c.interior(sol.w_aux[c.J("T")]), c.interior(sol.w_aux[c.J("P")])]


def run(state):
    case, s = state
    kind = case["kind"]
    if kind in ("turb", "cell"):
        s.step()
        return _fields(s)
    if kind in ("flame", "tube"):
        sol, graph = s
        sol.replay(graph)
        return _fields(sol)
    if kind == "rk53":
        s.rk_sync()
        return _fields(s)
    if kind == "reactors":
        br, T0, p0, Y0 = s
        out = br.integrate(T0, p0, Y0, case["t_max"], 1e-8, 1.05, 2.0, 20000, sync=False, order="coldest_first")
        return [out["Y"], out["T"], out["t_end"]]
    c = s.case
    if kind == "aux":
        s.compute_aux(1, 1)
        return [c.interior(s.w_aux[j]) for j in _aux_slots(c)]
    lib, ctx, st = s.lib, s.ctx, s.stream
    wa, fl = C.c_void_p(s.w_aux.data_ptr()), C.c_void_p(s.fl.data_ptr())
    check(lib.stx_euler_x(ctx, st, wa, fl, 1, c.nx, 1), "euler_x")
    check(lib.stx_euler_y(ctx, st, wa, fl, 1, c.ny, 0), "euler_y")
    check(lib.stx_euler_z(ctx, st, wa, fl, 1, c.nz, 0), "euler_z")
    check(lib.stx_visflx(ctx, st, wa, fl, 1), "visflx")
    check(lib.stx_visflx(ctx, st, wa, fl, 2), "visflx")
    return [s.fl[m] for m in range(c.nv)]


def _aux_slots(c):
    """w_aux as compute_aux writes it; the mixture fraction (constant here) left out."""
    return [j for j in range(2 * c.ns + 13) if j != c.J("Z")]


def work(case):
    """Bytes: the state in and out (and what the block writes).  Flops: per cell, from the
    method's formulas at nine species (recovery about 1.5e3, fluxes about 1.2e3 per
    direction, one chemistry right-hand side about 3e3)."""
    kind = case["kind"]
    ns = {"cell": 14, "rk53": 53, "flame": 11 if case.get("mech") == "flame_11sp" else 9}.get(kind, 9)
    n, steps = case.get("n", 0) ** 3, 1
    if kind in ("aux", "flux"):
        n = case["nx"] * case["ny"] * case["nz"]
    elif kind == "flame":
        n, steps = case["nx"], 10
    elif kind == "tube":
        n, steps = case["nx"] * case["ny"], case["steps"]
    elif kind == "cell":
        n = case.get("nx", 1) * case.get("ny", 1)
    if kind == "reactors":
        return {"bytes": 8.0 * case["n"] * (2 * 9 + 6), "flops": case["n"] * case["t_max"] / 1e-9 * 6 * 3e3}
    nv, q = ns + 4, (ns / 9.0) ** 2
    if kind == "aux":
        return {"bytes": 8.0 * n * (nv + 1 + 2 * ns + 14), "flops": 1.5e3 * n}
    if kind == "flux":
        return {"bytes": 8.0 * n * (2 * ns + 10 + nv), "flops": 3.6e3 * n}
    dirs = 3 if kind in ("turb", "rk53") else 1 + (case.get("ny", 1) > 1)
    flops = 3 * (1.5e3 * q + 1.2e3 * dirs * ns / 9.0)
    if kind != "rk53":
        flops += 10 * 3e3 * ns / 9.0 + 2 * 1.5e3 * q
    return {"bytes": 8.0 * n * steps * (2 * nv + 2 * ns + 14), "flops": flops * n * steps}


def tolerance(case):
    return TOLERANCE["split" if case.get("form") == "split" else case["kind"]]


# Measured spread between two evaluations whose inputs differ in their last bits (rel, max),
# and about four times that: aux 2e-15, 1e-13; flux 7e-14, 5e-12; rk53 4e-10, 2e-9; flame 1e-6,
# 2e-5; reactors 4e-5, 8e-4, with their basis in FP32 4e-3, 0.2.  The other steps show 5e-15
# where no cell changes its adaptive step count; one that does moves by 1e-7 or so, and the
# mixed form's fluxes round at 6e-8 of a step's change.
TOLERANCE = {
    "turb": {"rel": 1e-8, "max": 1e-5},
    "flame": {"rel": 5e-6, "max": 1e-4},
    "tube": {"rel": 1e-8, "max": 1e-5},
    "cell": {"rel": 1e-8, "max": 1e-5},
    "reactors": {"rel": 2e-4, "max": 4e-3},
    "split": {"rel": 1.6e-2, "max": 0.8},
    "aux": {"rel": 1e-14, "max": 5e-13},
    "flux": {"rel": 3e-13, "max": 2e-11},
    "rk53": {"rel": 2e-9, "max": 1e-8},
}


# ---------------------------------------------------------------- exact values, plain torch FP64
def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEV)


def _species_sum(tb, coef, T, Y, integral, const):
    """sum_k Y_k sum_l c_lk T^l (or its integral in T, plus the constant of integration)."""
    out = torch.zeros_like(T)
    for k in range(tb.ns):
        out = out + Y[k] * _species(tb, coef, T, k, integral, const)
    return out


def _species(tb, coef, T, k, integral, const):
    tr = tb.trange[k]
    m = torch.zeros(T.shape, dtype=torch.long, device=T.device)
    for q in range(1, tb.nsetcv):
        m = torch.where(T >= tr[q], q, m)
    cc = _t(coef[:, k, :])
    val = cc[tb.indx_cp_r + 1 - tb.indx_cp_l][m] if const else torch.zeros_like(T)
    for l in range(tb.indx_cp_l, tb.indx_cp_r + 1):
        a = cc[l - tb.indx_cp_l][m]
        if not integral:
            val = val + a * T ** l
        elif l == -1:
            val = val + a * torch.log(T)
        else:
            val = val + a / (l + 1.0) * T ** (l + 1)
    return val


def _energy(tb, T, Y):
    return _species_sum(tb, tb.cv_coeff, T, Y, True, True)


def _temperature(tb, e, Y, T):
    for _ in range(12):
        T = T + (e - _energy(tb, T, Y)) / _species_sum(tb, tb.cv_coeff, T, Y, False, False)
    return T


def _exact_aux(c, w, T0):
    """compute_aux of the interior: w and the guess T0 with ghosts; nine species."""
    tb, ns, ng = c.tb, c.ns, c.ng
    rY = w[:ns].clamp(min=0.0)
    rho = rY.sum(0)
    Y = rY / rho
    vel = [w[ns + m] / rho for m in range(3)]
    E = w[ns + 3] / rho
    e = E - 0.5 * sum(v * v for v in vel)
    core = (slice(ng, -ng),) * 3
    Yi, ri = Y[(slice(None),) + core], rho[core]
    T = _temperature(tb, e[core], Yi, T0[core])
    rg = _t(tb.rgas)
    rm = torch.einsum("k,kzyx->zyx", rg, Yi)
    cp = _species_sum(tb, tb.cp_coeff, T, Yi, False, False)
    p = ri * rm * T
    snd = torch.sqrt(cp / (cp - rm) * rm * T)
    x = (T - tb.t_min_tab) / tb.dt_tab
    it = x.long().clamp(0, tb.num_t_tab - 1)
    fr = x - it
    row = lambda a: _t(a)[it] + (_t(a)[it + 1] - _t(a)[it]) * fr
    mu_k, lam_k = [row(tb.visc[:, k]) for k in range(ns)], [row(tb.lam[:, k]) for k in range(ns)]
    X = Yi * (M.R_UNIV / rm) / _t(tb.mw)[:, None, None, None]
    lam = 0.5 * (sum(X[k] * lam_k[k] for k in range(ns)) + 1.0 / sum(X[k] / lam_k[k] for k in range(ns)))
    mu, rd = 0.0, []                    # the reference takes sqrt(mu_m / mu_l) in the Wilke factor
    for l in range(ns):
        den, inv = 0.0, 0.0
        for m in range(ns):
            rw = tb.mw[l] / tb.mw[m]
            den = den + X[m] * (1.0 + torch.sqrt(mu_k[m] / mu_k[l]) * rw ** -0.25) ** 2 / math.sqrt(8.0 * (1.0 + rw))
            if m != l:
                inv = inv + X[m] / row(tb.diffbin[:, l, m])
        mu = mu + X[l] * mu_k[l] / den
        rd.append((1.0 - Yi[l]) / inv * c.p0 / p * ri)
    # gradients, dilatation / 3 and the Ducros sensor (sensor_type 1)
    grad = [[_deriv(c, v, d) for d in range(3)] for v in vel]
    div = grad[0][0] + grad[1][1] + grad[2][2]
    om = (grad[2][1] - grad[1][2]) ** 2 + (grad[0][2] - grad[2][0]) ** 2 + (grad[1][0] - grad[0][1]) ** 2
    duc = (-div / torch.sqrt(om + div * div + c.eps_sensor)).clamp(min=0.0) ** 2
    h = E[core] + p / ri
    out = list(Yi) + [v[core] for v in vel] + [h, T, p, snd, mu, duc, div / 3.0, ri, lam] + rd
    return out


_CD = (0.75, -0.15, 1.0 / 60.0)


def _shift(a, c, d, s):
    """Interior of a moved by s cells along direction d (0: x)."""
    ng = c.ng
    sl = [slice(ng, a.shape[q] - ng) for q in range(3)]
    q = 2 - d
    sl[q] = slice(ng + s, a.shape[q] - ng + s)
    return a[tuple(sl)]


def _metric(c, d):
    m = _t((c.dcsidx, c.detady, c.dzitdz)[d])
    return m.reshape([-1 if q == 2 - d else 1 for q in range(3)])


def _deriv(c, a, d):
    return sum(cf * (_shift(a, c, d, l + 1) - _shift(a, c, d, -l - 1)) for l, cf in enumerate(_CD)) * _metric(c, d)


def _keep(f, un):
    """KEEP(2) face flux of order 6; f: fields of shape (6, faces), slots -2..3 around the face."""
    def fac(a, b, energy):
        t = ((b - a) / (a + b)) ** 2
        s = 1.0 + t / 3.0 + t * t / 5.0
        return s / (1.0 + t + t * t) if energy else 1.0 / s

    out = [0.0] * (len(f["Y"]) + 4)
    ns = len(f["Y"])
    e = f["h"] - f["p"] / f["r"] - 0.5 * sum(v * v for v in f["v"])
    for l in range(1, 4):
        for m in range(l):
            a, b = 2 - m, 2 - m + l
            r, v = f["r"], f["v"]
            q = (v[un][a] + v[un][b]) * (r[a] + r[b]) * fac(r[a], r[b], False) * _CD[l - 1]
            for k in range(ns):
                out[k] = out[k] + 0.25 * q * (f["Y"][k][a] + f["Y"][k][b])
            for d in range(3):
                out[ns + d] = out[ns + d] + 0.25 * q * (v[d][a] + v[d][b])
            out[ns + un] = out[ns + un] + _CD[l - 1] * (f["p"][a] + f["p"][b])
            out[ns + 3] = out[ns + 3] + 0.25 * (
                q * (e[a] + e[b]) * fac(e[a], e[b], True) + q * sum(x[a] * x[b] for x in v) +
                _CD[l - 1] * 4.0 * (v[un][a] * f["p"][b] + v[un][b] * f["p"][a]))
    return torch.stack(out)


def _weno5z(vp, bs):
    """WENO5-Z value at the face right of slot 2 of vp (5, ...)."""
    a, b, c, d, e = vp
    d0, d1 = 13.0 / 12.0, 0.25
    be = [bs * (d0 * (c - 2 * b + a) ** 2 + d1 * (3 * c - 4 * b + a) ** 2),
          bs * (d0 * (b - 2 * c + d) ** 2 + d1 * (b - d) ** 2),
          bs * (d0 * (c - 2 * d + e) ** 2 + d1 * (3 * c - 4 * d + e) ** 2)]
    tau = (be[0] - be[2]).abs() + 1e-40
    w = [g * (x + tau) / (x + 1e-40) for g, x in zip((0.1, 0.6, 0.3), be)]
    q = [(2 * a - 7 * b + 11 * c) / 6.0, (-b + 5 * c + 2 * d) / 6.0, (2 * c + 5 * d - e) / 6.0]
    return sum(x * y for x, y in zip(w, q)) / sum(w)


def _weno(c, f, un):
    """Characteristic WENO5-Z flux with local Lax-Friedrichs splitting on the Roe state."""
    tb, ns = c.tb, c.ns
    rg = _t(tb.rgas)
    L, R = 2, 3
    r, v, h, p, Y = f["r"], f["v"], f["h"], f["p"], f["Y"]
    ek = 0.5 * sum(x * x for x in v)
    e = h - p / r - ek
    s = torch.sqrt(r[R] / r[L])
    avg = lambda q: (s * q[R] + q[L]) / (s + 1.0)
    rr, va, ha, ea = s * r[L], [avg(x) for x in v], avg(h), avg(e)
    ya = torch.stack([avg(Y[k]) for k in range(ns)])
    kin = 0.5 * sum(x * x for x in va)
    por = ha - ea - kin
    rm = torch.einsum("k,kf->f", rg, ya)
    T = _temperature(tb, ea, ya, por / rm)
    cp = _species_sum(tb, tb.cp_coeff, T, ya, False, False)
    gm1 = cp / (cp - rm) - 1.0
    pe = rr * gm1
    pr = torch.stack([rg[k] * T + gm1 * (ea - _species(tb, tb.cv_coeff, T, k, True, True)) for k in range(ns)])
    drho = torch.stack([r[R] * Y[k][R] - r[L] * Y[k][L] for k in range(ns)])
    de, dp = e[R] - e[L], p[R] - p[L]
    pede = pe * de
    err = dp - pede - (pr * drho).sum(0)
    fac = err / (pede * pede + ((pr * drho) ** 2).sum(0)).clamp(min=1e-6)
    pe = pe * (1.0 + pede * fac)
    pr = pr * (1.0 + pr * drho * fac)
    cc = por / rr * pe + (ya * pr).sum(0)
    cs = torch.sqrt(cc)
    b3 = ea + kin
    b2 = pe / (rr * cc)
    b1 = -b2 * (b3 - 2.0 * kin) + pr / cc
    t1, t2 = [d for d in range(3) if d != un]
    # conserved variables and fluxes of the stencil, (6, faces)
    ru = r * v[un]
    W = [r * Y[k] for k in range(ns)] + [r * x for x in v] + [r * h - p]
    G = [ru * Y[k] for k in range(ns)] + [ru * x for x in v] + [ru * h]
    G[ns + un] = G[ns + un] + p
    ev = [(v[un] - f["c"]).abs().amax(0), v[un].abs().amax(0), (v[un] + f["c"]).abs().amax(0)]

    def project(q):
        Q = sum(b1[k] * q[k] for k in range(ns)) + b2 * (q[ns + 3] - sum(va[d] * q[ns + d] for d in range(3)))
        S = sum(q[k] for k in range(ns))
        a = (va[un] * S - q[ns + un]) / cs
        return ([0.5 * (Q + a)] + [q[k] - ya[k] * Q for k in range(ns)] +
                [q[ns + t1] - va[t1] * S, q[ns + t2] - va[t2] * S, 0.5 * (Q - a)])

    cw, cg = project(W), project(G)
    r2u2 = c.rho0 ** 2 * c.u0 ** 2
    fi = []
    for m in range(ns + 4):
        lam = ev[0] if m == 0 else (ev[2] if m == ns + 3 else ev[1])
        bs = 1.0 / (r2u2 * c.u0 ** 2) if m in (ns + 1, ns + 2) else 1.0 / r2u2
        vp = 0.5 * (cg[m] + lam * cw[m])
        vm = cg[m] - vp
        fi.append(_weno5z(vp[0:5], bs) + _weno5z(vm.flip(0)[0:5], bs))
    f0, f4, g1, g2 = fi[0], fi[ns + 3], fi[ns + 1], fi[ns + 2]
    fs = torch.stack(fi[1:ns + 1])
    tot = f0 + f4 + fs.sum(0)
    out = [ya[k] * (f0 + f4) + fs[k] for k in range(ns)] + [None] * 4
    out[ns + un] = va[un] * tot + cs * (f4 - f0)
    out[ns + t1] = va[t1] * tot + g1
    out[ns + t2] = va[t2] * tot + g2
    out[ns + 3] = (ha * (f0 + f4) + va[un] * cs * (f4 - f0) + ((b3 - pr / (b2 * cc)) * fs).sum(0) +
                   va[t1] * g1 + va[t2] * g2)
    return torch.stack(out)


def _convective(c, wa, d):
    """Hybrid flux divergence along direction d, (nv, nz, ny, nx)."""
    ns, ng, n = c.ns, c.ng, (c.nx, c.ny, c.nz)[d]
    q = 3 - d
    sl = [slice(None)] + [slice(ng, wa.shape[x] - ng) if x != q else slice(None) for x in (1, 2, 3)]
    a = wa[tuple(sl)].movedim(q, -1)                          # (field, lateral, lateral, sweep)
    flat = lambda j: torch.stack([a[j][..., ng - 3 + s:ng - 3 + s + n + 1].reshape(-1) for s in range(6)])
    J = c.J
    f = dict(Y=[flat(k) for k in range(ns)], v=[flat(J("U") + m) for m in range(3)], h=flat(J("H")), p=flat(J("P")),
             r=flat(J("R")), c=flat(J("C")))
    hat = _keep(f, d)
    shock = (flat(J("DUC")) > c.sensor_threshold).any(0)
    if shock.any():
        pick = lambda x: [y[:, shock] for y in x] if isinstance(x, list) else x[:, shock]
        hat[:, shock] = _weno(c, {k: pick(x) for k, x in f.items()}, d)
    hat = hat.reshape((c.nv,) + a.shape[1:3] + (n + 1,))
    return ((hat[..., 1:] - hat[..., :-1]) * _t((c.dcsidx, c.detady, c.dzitdz)[d])).movedim(-1, q)


def _viscous(c, wa, d):
    """Staggered viscous, heat and species-diffusion flux divergence along direction d."""
    tb, ns, ng, n = c.tb, c.ns, c.ng, (c.nx, c.ny, c.nz)[d]
    q = 3 - d
    sl = [slice(None)] + [slice(ng, wa.shape[x] - ng) if x != q else slice(None) for x in (1, 2, 3)]
    a = wa[tuple(sl)].movedim(q, -1)
    J = c.J
    x = _t((c.x, c.y, c.z)[d])
    dx = x[ng:ng + n + 1] - x[ng - 1:ng + n]
    lo = lambda b: b[..., ng - 1:ng + n]
    hi = lambda b: b[..., ng:ng + n + 1]
    mean = lambda b: 0.5 * (lo(b) + hi(b))
    jump = lambda b: (hi(b) - lo(b)) / dx
    vel = [a[J("U") + m] for m in range(3)]
    mu, lam = mean(a[J("MU")]), mean(a[J("K_COND")])
    Y = [a[k] for k in range(ns)]
    wm = M.R_UNIV / sum(float(tb.rgas[k]) * Y[k] for k in range(ns))
    rmean = 0.5 * (lo(wm) + hi(wm)) / (lo(wm) * hi(wm))
    jk = [mean(a[J("K_COND") + 1 + k]) * jump(Y[k] * wm) * rmean for k in range(ns)]
    tot = sum(jk)
    spec = [-jk[k] + tot * mean(Y[k]) for k in range(ns)]
    T = a[J("T")]
    he = sum(spec[k] * mean(_species(tb, tb.cp_coeff, T, k, True, True)) for k in range(ns))
    heat = lam * jump(T) + mu * jump(0.5 * sum(v * v for v in vel))
    hat = torch.stack(spec + [-mu * jump(v) for v in vel] + [he - heat])
    w = 2.0 / (x[ng + 1:ng + n + 1] - x[ng - 1:ng + n - 1])
    return ((hat[..., 1:] - hat[..., :-1]) * w).movedim(-1, q)


def _collocated(c, wa):
    """The cross and dilatation terms of the viscous stress, added to the momentum and energy rows."""
    J, i = c.J, c.interior
    vel = [wa[J("U") + m] for m in range(3)]
    mu, th = wa[J("MU")], wa[J("DIV")]
    g = [[_deriv(c, v, d) for d in range(3)] for v in vel]                  # g[m][d] = d v_m / d x_d
    dmu, dth = [_deriv(c, mu, d) for d in range(3)], [_deriv(c, th, d) for d in range(3)]
    s = [[g[d][m] - (2.0 * i(th) if m == d else 0.0) for d in range(3)] for m in range(3)]
    sig = [sum(dmu[d] * s[m][d] for d in range(3)) + i(mu) * dth[m] for m in range(3)]
    work_ = i(mu) * sum(s[m][d] * g[m][d] for m in range(3) for d in range(3))
    return sig + [sum(sig[m] * i(vel[m]) for m in range(3)) + work_]


def exact(case, seed):
    if case["kind"] not in ("aux", "flux"):
        return None
    _, s = prepare(case, seed)
    c = s.case
    if case["kind"] == "aux":
        return _exact_aux(c, s.w, s.w_aux[c.J("T")])
    fl = torch.zeros_like(s.fl)
    for d in range(3):
        fl += _convective(c, s.w_aux, d) + _viscous(c, s.w_aux, d)
    for m, x in enumerate(_collocated(c, s.w_aux)):
        fl[c.ns + m] -= x
    return [fl[m] for m in range(c.nv)]
