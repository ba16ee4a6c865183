"""The work that programs have this framework do, as timeable cases.

Each case names a path (`work`), a box, a precision and a flow; `prepare`
builds the seeded flow and the operator a program keeps, `run` makes one pass
through the public entry points, and `exact` evaluates the same pass in plain
torch, in 64 bits, from the equations: the Valencia scheme on an analytic (or
grid-held) metric, with MUSCL reconstruction, the HLLE flux and the bracketed
Newton recovery of the primitives."""
from __future__ import annotations

import math

import torch

import grdzhadzha_b200 as G
from grdzhadzha_b200 import workloads as W
from grdzhadzha_b200.adjoint import TorusAccretionAdjoint, default_torus
from grdzhadzha_b200.ensemble import Ensemble
from grdzhadzha_b200.operator import (LevelBox, LevelDataFiniteVolumeOperator,
                                      kitp_config)

CFL = 0.25
# a program restarts its flow from the initial state after so many steps
# (the length of the framework's runs: 100 to 400 steps)
RUN_STEPS = 100
# floating-point operations of one right-hand side of a cell: three faces of
# about 400, the recovery, the metric and the sources
RHS_FLOPS = 1600.0


def listed():
    return [
        # one patch of a level, the smallest a mesh hands out: the hooks call
        # the right-hand side patch by patch
        dict(name="rhs patch 16", work="rhs", flow="torus", precision="fp64",
             nx=16, ny=16, nz=16),
        # a ragged patch on the moving binary's metric (volume-time source)
        dict(name="rhs binary 45x38x31", work="rhs", flow="binary",
             precision="fp64", nx=45, ny=38, nz=31),
        # spherical accretion at its usual size, the accretion rate read
        # after every step
        dict(name="rk4 michel 64", work="rk4", flow="michel",
             precision="fp64", nx=64, ny=64, nz=64, steps=1),
        # the torus runs: FP64, and mixed precision
        dict(name="rk4 torus 256", work="rk4", flow="torus",
             precision="fp64", nx=256, ny=256, nz=256, steps=2),
        dict(name="rk4 torus 256 mixed", work="rk4", flow="torus",
             precision="mixed", nx=256, ny=256, nz=256, steps=2),
        # the circumbinary disk, the largest grid
        dict(name="rk4 disk 320 mixed", work="rk4", flow="disk",
             precision="mixed", nx=320, ny=320, nz=320, steps=1),
        # a level of eight boxes with ghost exchange, SSPRK2
        dict(name="level 8 boxes", work="level", flow="torus",
             precision="fp64", nx=130, ny=114, nz=96, boxes=8),
        # the metric held by the grid (CCZ4 variables), SSPRK2
        dict(name="ccz4 100x90x70", work="ccz4", flow="torus",
             precision="fp64", nx=100, ny=90, nz=70),
        # the disk driver's step: viscosity, sinks, SSPRK2
        dict(name="kitp 128x128x48", work="kitp", flow="disk",
             precision="fp64", nx=128, ny=128, nz=48),
        # many independent flows of uneven size in one launch
        dict(name="ensemble 24 mixed", work="ensemble", flow="mixture",
             precision="mixed", members=24, nmin=32, nmax=96, steps=2),
        # a level that the host keeps in its own memory
        dict(name="host step 161x143x127", work="host", flow="torus",
             precision="fp64", nx=161, ny=143, nz=127),
        # the gradient of the accreted mass, forward and backward
        dict(name="adjoint 64", work="adjoint", flow="torus",
             precision="fp64", nx=64, ny=64, nz=64, steps=4),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    work = rng.choice(["rhs", "rhs", "rk4", "rk4", "rk4", "level", "ccz4",
                       "kitp", "ensemble", "host", "adjoint"])
    c = dict(work=work, flow="torus", precision="fp64")
    lo, hi = dict(rhs=(14, 128), rk4=(32, 256), level=(40, 150),
                  ccz4=(24, 110), kitp=(40, 150), host=(40, 170),
                  adjoint=(28, 72), ensemble=(32, 96))[work]
    if work == "ensemble":
        c.update(flow="mixture", precision=rng.choice(["fp64", "mixed"]),
                 members=_size(rng, 4, 24), nmin=rng.choice([24, 32, 40]),
                 nmax=rng.choice([48, 64, 80, 96]), steps=rng.choice([1, 2]))
        return c
    n = _size(rng, lo, hi)
    c.update(nx=n, ny=max(lo, int(n * rng.uniform(0.75, 1.0))),
             nz=max(lo, int(n * rng.uniform(0.6, 1.0))))
    if work == "rhs":
        c["flow"] = rng.choice(["torus", "binary", "michel"])
    elif work == "rk4":
        c.update(flow=rng.choice(["torus", "michel", "disk"]),
                 precision=rng.choice(["fp64", "mixed"]),
                 steps=rng.choice([1, 2]))
    elif work == "level":
        c["boxes"] = rng.choice([1, 2, 4, 8])
    elif work == "kitp":
        c["flow"] = "disk"
    elif work == "host":
        c["precision"] = rng.choice(["fp64", "mixed"])
    elif work == "adjoint":
        c["steps"] = rng.choice([2, 4, 6])
    return c


# ------------------------------------------------------------- the programs


def _flow(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    p = case["precision"]
    if case["flow"] == "michel":
        return W.michel(n, seed=seed, accretion_radius=4.0, precision=p)
    if case["flow"] == "binary":
        op, lv = W.binary_pn_disk(n, precision=p)
        op.perturb_density(lv, 1e-3, seed)
        op.recover_primitives(lv)
        return op, lv
    if case["flow"] == "disk":
        return W.binary_disk(n, seed=seed, precision=p)
    if case["work"] == "rhs":
        return _torus_patch(n, seed, p)
    return W.kerr_schild_torus(n, seed=seed, precision=p)


def _torus_patch(n, seed, precision):
    """A patch of n cells beside the hole, inside a larger torus grid: its
    ghosts hold the neighbours' cells."""
    N = max(64, 3 * max(n) // 2)
    op, lv = W.kerr_schild_torus(N, seed=seed, precision=precision)
    x, y, z = (3 * (N - n[0]) // 4, (N - n[1]) // 2, (N - n[2]) // 2)
    return op, LevelBox(
        lo=(x, y, z), hi=(x + n[0] - 1, y + n[1] - 1, z + n[2] - 1),
        domain_lo=lv.lo, domain_hi=lv.hi,
        state=lv.state[:, z:z + n[2] + 4, y:y + n[1] + 4,
                       x:x + n[0] + 4].clone())


def _cut(n, parts):
    """Half-open spans that cut n cells as evenly as they can."""
    e = [n * q // parts for q in range(parts + 1)]
    return list(zip(e, e[1:]))


def _level_boxes(lv, boxes):
    """The box `lv` of the whole domain cut into `boxes` (1, 2, 4 or 8)."""
    cuts = {1: (1, 1, 1), 2: (1, 1, 2), 4: (1, 2, 2), 8: (2, 2, 2)}[boxes]
    nx, ny, nz = (lv.hi[d] + 1 for d in range(3))
    out = []
    for z0, z1 in _cut(nz, cuts[2]):
        for y0, y1 in _cut(ny, cuts[1]):
            for x0, x1 in _cut(nx, cuts[0]):
                out.append(LevelBox(
                    lo=(x0, y0, z0), hi=(x1 - 1, y1 - 1, z1 - 1),
                    domain_lo=lv.lo, domain_hi=lv.hi,
                    state=lv.state[:, z0:z1 + 4, y0:y1 + 4,
                                   x0:x1 + 4].clone()))
    return out


def prepare(case, seed):
    work = case["work"]
    if work == "ensemble":
        members = _members(case, seed)
        start = [lv.state.clone() for _, lv in members]
        return dict(case=case, members=members, start=start, done=0,
                    ens=Ensemble(members, cfl=CFL))
    if work == "adjoint":
        return _prepare_adjoint(case, seed)
    op, lv = _flow(case, seed)
    s = dict(case=case, op=op, lv=lv, inv=[1.0 / op.dx] * 3, done=0, t=0.0,
             mi=0.0)
    if work == "rhs":
        s["rhs"] = lv.new_rhs()
        return s
    if work == "level":
        s["boxes"] = _level_boxes(lv, case["boxes"])
        s["stages"] = [LevelBox(lo=b.lo, hi=b.hi, domain_lo=b.domain_lo,
                                domain_hi=b.domain_hi) for b in s["boxes"]]
        del s["lv"]
        s["start"] = [b.state.clone() for b in s["boxes"]]
    elif work == "ccz4":
        s["lv"] = op.ccz4_state(lv)
        p = op.params
        s["cop"] = LevelDataFiniteVolumeOperator(
            op.eos, G.AtmosphereOptions(p.rho_floor, p.pressure_floor,
                                        p.max_velocity_squared),
            p.limiter_theta, True,
            G.RecoveryOptions(p.recovery_max_iterations,
                              p.recovery_tolerance,
                              p.recovery_pressure_floor,
                              p.recovery_max_velocity_squared))
        s["start"] = [s["lv"].state.clone()]
    elif work == "host":
        s["host"] = lv.state.cpu().pin_memory()
        s["mi"] = op.compute_max_inverse_dt(lv)
        s["start"] = [lv.state.cpu()]
    else:
        s["start"] = [lv.state.clone()]
    if work == "kitp":
        s["cfg"] = kitp_config()
    return s


def _member_sizes(case):
    """Uneven sizes spread over nmin..nmax, odd ones among them."""
    span = case["nmax"] - case["nmin"] + 1
    return [case["nmin"] + 29 * i % span for i in range(case["members"])]


def _members(case, seed):
    """Half Michel inflows, half tori, their parameters from the seed
    (batched_ensemble's ranges)."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for i, n in enumerate(_member_sizes(case)):
        u = torch.rand(3, generator=gen, dtype=torch.float64).tolist()
        p = case["precision"]
        if i < case["members"] // 2:
            rs = 5.0 + 7.0 * u[0]
            out.append(W.michel(n, sonic_radius=rs, half_width=2.0 * rs,
                                seed=seed + i, accretion_radius=4.0,
                                precision=p))
        else:
            rin = 6.0 + 4.0 * u[0]
            out.append(W.kerr_schild_torus(
                n, spin=0.99 * u[1], gamma=(4.0 if u[2] < 0.5 else 5.0) / 3.0,
                inner_radius=rin, pressure_max_radius=rin + 6.0,
                seed=seed + i, accretion_radius=2.5, precision=p))
    return out


def _prepare_adjoint(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    gen = torch.Generator().manual_seed(seed)
    u = torch.rand(6, generator=gen, dtype=torch.float64).tolist()
    spin = 0.6 + 0.2 * u[5]
    dx = 40.0 / n[0]
    op = G.TimeDependentFixedBGLevelDataFiniteVolumeOperator(
        G.IdealGasEOS(5.0 / 3.0), G.KerrSchild(mass=1.0, spin=spin, dx=dx),
        dx, tuple(0.5 * m * dx for m in n),
        G.AtmosphereOptions(1e-10, 1e-12, 0.8), 2.0, True,
        G.RecoveryOptions(80, 1e-12, 1e-12, 0.9), True, False, 1e-3, 1.5,
        5.0, "fp64")
    lv = LevelBox.cube(n)
    torus = default_torus(spin=spin, mode_amplitude=[1e-2, 8e-3, 6e-3, 4e-3,
                                                     2e-3],
                          mode_phase=[2.0 * math.pi * x for x in u[:5]])
    probe = TorusAccretionAdjoint(op, lv, 1, 1, 1.0, torus)
    probe.initial_state(level=lv)
    dt = CFL / op.compute_max_inverse_dt(lv)
    del probe
    every = max(1, case["steps"] // 2)
    adj = TorusAccretionAdjoint(op, lv, case["steps"], every, dt, torus)
    return dict(case=case, op=op, lv=lv, adj=adj, dt=dt)


def _restart(s, states, steps):
    """Begins the run again when its steps are done."""
    if s["done"] >= RUN_STEPS:
        for x, x0 in zip(states, s["start"]):
            x.copy_(x0)
        s["done"], s["t"], s["mi"] = 0, 0.0, 0.0
        if "ens" in s:
            s["ens"].invalidate()
    s["done"] += steps


def run(s):
    case = s["case"]
    work = case["work"]
    if work == "rhs":
        s["op"].compute_rhs(s["rhs"], s["lv"], None, s["inv"])
        return s["rhs"]
    if work == "adjoint":
        J = s["adj"].forward()
        return dict(J=J, grad=torch.tensor(s["adj"].backward(),
                                           dtype=torch.float64))
    if work == "ensemble":
        _restart(s, [lv.state for _, lv in s["members"]], case["steps"])
        s["ens"].advance(case["steps"])
        return [lv.interior() for _, lv in s["members"]]
    if work == "level":
        _restart(s, [b.state for b in s["boxes"]], 1)
        op, boxes = s["op"], s["boxes"]
        dt = min(op.compute_stable_dt(b, None, s["inv"], CFL) for b in boxes)
        if len(boxes) == 1:
            op.advance_ssprk2(boxes[0], None, s["inv"], 0.0, dt)
        else:
            op.advance_level_ssprk2(boxes, s["stages"], dt, s["inv"])
        return [b.interior() for b in boxes]
    if work == "host":
        _restart(s, [s["host"]], 1)
        dt, s["mi"], *_ = s["op"].advance_rk4_cfl_host(
            s["host"], s["lv"], CFL, s["t"], 0.0, s["mi"], s["inv"])
        s["t"] += dt
        z, y, x = s["lv"].interior_shape
        return s["host"][:, 2:2 + z, 2:2 + y, 2:2 + x]
    lv = s["lv"]
    _restart(s, [lv.state], case.get("steps", 1))
    if work == "ccz4":
        dt = s["cop"].compute_stable_dt(lv, None, s["inv"], CFL)
        s["cop"].advance_ssprk2(lv, None, s["inv"], dt)
        return lv.interior(slice(25, 36))
    if work == "kitp":
        dt = s["op"].compute_stable_dt(lv, None, s["inv"], CFL, s["t"])
        s["op"].kitp_advance_ssprk2(lv, s["t"], dt, s["cfg"], s["inv"])
        s["t"] += dt
        return lv.interior()
    if case["steps"] > 1:
        s["t"], s["mi"], _ = s["op"].advance_rk4_cfl_steps(
            lv, CFL, case["steps"], s["t"], 0.0, s["mi"], s["inv"])
    else:
        dt, s["mi"], _ = s["op"].advance_rk4_cfl(lv, CFL, s["t"], 0.0,
                                                 s["mi"], s["inv"])
        s["t"] += dt
    out = dict(state=lv.interior(), next_max_inverse_dt=s["mi"])
    if case["flow"] == "michel":
        out["mdot"] = s["op"].accretion()[0]
    return out


def work(case):
    if case["work"] == "ensemble":
        cells = sum(m ** 3 for m in _member_sizes(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    steps = case.get("steps", 1)
    # right-hand sides, values read and values written of a pass
    rhs, inp, out = dict(
        rhs=(1, 5, 5), rk4=(4 * steps, 5, 11), ensemble=(4 * steps, 5, 11),
        level=(2, 5, 11), ccz4=(2, 27, 11), kitp=(2, 5, 11), host=(4, 5, 11),
        # forward sweep, and its reverse at twice that
        adjoint=(12 * steps, 0, 0))[case["work"]]
    # the adjoint cannot do without the states of its steps
    bytes_ = 8.0 * cells * (inp + out + (10 * steps if
                                         case["work"] == "adjoint" else 0))
    return dict(bytes=bytes_, flops=RHS_FLOPS * rhs * cells)


# ------------------------------------------- the equations in plain torch
# A symmetric 3x3 tensor is a list of six fields (00 01 02 11 12 22); the
# fields of a box include its two ghost cells on each side, (z, y, x).

_SYM = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
_PAIR = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]


def _det(g):
    return (g[0] * (g[3] * g[5] - g[4] * g[4])
            - g[1] * (g[1] * g[5] - g[4] * g[2])
            + g[2] * (g[1] * g[4] - g[3] * g[2]))


def _inverse(g):
    d = _det(g)
    return [(g[3] * g[5] - g[4] * g[4]) / d, (g[2] * g[4] - g[1] * g[5]) / d,
            (g[1] * g[4] - g[2] * g[3]) / d, (g[0] * g[5] - g[2] * g[2]) / d,
            (g[1] * g[2] - g[0] * g[4]) / d, (g[0] * g[3] - g[1] * g[1]) / d]


def _lower(g, v):
    return [sum(g[_SYM[i][j]] * v[j] for j in range(3)) for i in range(3)]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _ks(p):
    """(x, y, z, t) -> gamma_ij, lapse, shift of the Kerr-Schild hole."""
    M, a = p.ks_mass, p.ks_spin

    def metric(x, y, z, t):
        rho2 = torch.clamp(torch.sqrt(x * x + y * y + z * z), min=1e-6) ** 2
        A = rho2 - a * a
        r2 = 0.5 * A + torch.sqrt(0.25 * A * A + a * a * z * z)
        r = torch.sqrt(r2)
        ct = z / r
        H2 = 2.0 * M * r / (r2 + a * a * ct * ct)
        el = [(r * x + a * y) / (r2 + a * a), (r * y - a * x) / (r2 + a * a),
              ct]
        gam = [(1.0 if i == j else 0.0) + H2 * el[i] * el[j]
               for i, j in _PAIR]
        c = H2 / (1.0 + H2 * _dot(el, el))
        return tuple(gam) + (1.0 / torch.sqrt(1.0 + H2),) + tuple(
            c * e for e in el)
    return metric


def _orbit(p, t):
    """Positions and velocities of the binary's bodies at time t."""
    total = p.pn_mass_1 + p.pn_mass_2
    om = p.pn_angular_velocity or math.sqrt(total / p.pn_separation ** 3)
    ph = p.pn_phase + om * (p.pn_time + t)
    out = []
    for m, sgn in ((p.pn_mass_2, 1.0), (p.pn_mass_1, -1.0)):
        r = sgn * m / total * p.pn_separation
        out.append(((r * math.cos(ph), r * math.sin(ph), 0.0),
                    (-om * r * math.sin(ph), om * r * math.cos(ph), 0.0)))
    return out, om


def _pn(p, t0):
    """(x, y, z, t) -> metric of the binary whose bodies move on straight
    lines from their places and velocities at t0."""
    bodies, _ = _orbit(p, t0)
    soft2 = p.pn_softening_radius ** 2

    def metric(x, y, z, t):
        U, V = 0.0, [0.0, 0.0, 0.0]
        for m, (pos, vel) in zip((p.pn_mass_1, p.pn_mass_2), bodies):
            d = [q - pos[i] - vel[i] * t for i, q in enumerate((x, y, z))]
            u = m / torch.sqrt(soft2 + _dot(d, d))
            U = U + u
            V = [V[i] + vel[i] * u for i in range(3)]
        psi = 1.0 + 2.0 * U
        lapse = torch.sqrt(1.0 - 2.0 * U + 2.0 * U * U
                           + 16.0 * _dot(V, V) / psi)
        zero = torch.zeros_like(psi)
        return (psi, zero, zero, psi, zero, psi, lapse) + tuple(
            -4.0 * v / psi for v in V)
    return metric


class _Geometry:
    """Metric of every ghosted cell of a box and its derivatives."""

    def __init__(self, p, glo, shape, t):
        dev = torch.device("cuda")
        ax = [(torch.arange(shape[2 - d], device=dev, dtype=torch.float64)
               + (glo[d] + 0.5)) * p.dx - p.center[d] for d in range(3)]
        z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        x, y, z = x.contiguous(), y.contiguous(), z.contiguous()
        self.pos = [x, y, z]
        binary = p.background == 1
        f = _pn(p, t) if binary else _ks(p)
        zero, one = torch.zeros_like(x), torch.ones_like(x)
        args = (x, y, z, zero)
        val = f(*args)
        self.gLL, self.lapse, self.shift = list(val[:6]), val[6], val[7:]
        self.gUU = _inverse(self.gLL)
        dgam, self.dlapse, dshift = [], [], []
        for d in range(3):
            dv = torch.func.jvp(f, args, tuple(
                one if q == d else zero for q in range(4)))[1]
            dgam.append(dv[:6])
            self.dlapse.append(dv[6])
            dshift.append(dv[7:])
        dt_gam = None
        if binary:
            dt_gam = torch.func.jvp(f, args, (zero, zero, zero, one))[1][:6]
        self.dgam = dgam
        self.dshift = dshift  # [direction][component]
        self.dlnsqrtg = [0.5 * _trace(self.gUU, dgam[d]) for d in range(3)]
        self.K = []
        for q, (i, j) in enumerate(_PAIR):
            k = _dot(self.shift, [dgam[m][q] for m in range(3)])
            for m in range(3):
                k = k + self.gLL[_SYM[m][j]] * dshift[i][m] \
                    + self.gLL[_SYM[m][i]] * dshift[j][m]
            if binary:
                k = k - dt_gam[q]
            self.K.append(k / (2.0 * self.lapse))
        r = torch.sqrt(x * x + y * y + z * z)
        self.excised = r < p.excision_radius
        self.inside = r < p.accretion_radius
        self.volume_rate = None
        if binary and p.use_metric_volume_time_sources:
            # central difference in time of ln sqrt(det gamma)
            h = max(p.metric_time_derivative_step, 1e-12)
            lnd = [0.5 * torch.log(_pn(p, t + q)(*args)[0] ** 3)
                   for q in (h, -h)]
            self.volume_rate = (lnd[0] - lnd[1]) / (2.0 * h)


def _trace(a, b):
    return sum((1.0 if i == j else 2.0) * a[q] * b[q]
               for q, (i, j) in enumerate(_PAIR))


def _p2c(pr, gLL):
    rho, p, v, eps = pr
    vL = _lower(gLL, v)
    W2 = 1.0 / (1.0 - _dot(vL, v))
    rhw = rho * (1.0 + eps + p / rho) * W2
    D = rho * torch.sqrt(W2)
    return [D, rhw * vL[0], rhw * vL[1], rhw * vL[2], rhw - p - D]


def _eps(o, rho, p):
    return p / ((o.adiabatic_index - 1.0) * rho)


def _floors(o, rho, p, v, gLL):
    rho = torch.clamp(rho, min=o.rho_floor)
    p = torch.clamp(p, min=o.pressure_floor)
    v2 = _dot(_lower(gLL, v), v)
    cap = o.max_velocity_squared
    f = torch.where(v2 >= cap, torch.sqrt(cap / v2), torch.ones_like(v2))
    return rho, p, [f * q for q in v], _eps(o, rho, p)


def _con2prim(o, U, gUU):
    """The bracketed Newton recovery: the first iterate whose residual is
    below the tolerance.  Returns ((rho, p, v), recovered)."""
    D, S, tau = U[0], U[1:4], U[4]
    Gf = o.adiabatic_index / (o.adiabatic_index - 1.0)
    mom = _lower(gUU, S)
    S2 = _dot(mom, S)
    tol, cap = o.recovery_tolerance, o.recovery_max_velocity_squared

    def residual(p):
        e = tau + D + p
        v2 = torch.clamp(S2 / (e * e), max=cap)
        Wl = 1.0 / torch.sqrt(1.0 - v2)
        dW = -Wl ** 3 * v2 / e
        return (D * Wl + Gf * p * Wl * Wl - e,
                D * dW + Gf * (Wl * Wl + 2.0 * p * Wl * dW) - 1.0)

    lower = torch.full_like(D, o.recovery_pressure_floor)
    f_lower = residual(lower)[0]
    ok = (D > 0.0) & ~((f_lower >= 0.0) & (f_lower.abs() > tol))
    neg = f_lower < 0.0
    upper = torch.where(neg, torch.clamp(tau.abs() + D, min=1.0), lower)
    for _ in range(o.recovery_max_iterations):
        grow = neg & (residual(upper)[0] <= 0.0)
        if not bool(grow.any()):
            break
        upper = torch.where(grow, 2.0 * upper, upper)
    p = torch.where(f_lower.abs() <= tol, lower, torch.minimum(
        torch.maximum(tau * (o.adiabatic_index - 1.0), lower), upper))
    r, dr = residual(p)
    for _ in range(o.recovery_max_iterations):
        go = ok & ~(r.abs() < tol)
        if not bool(go.any()):
            break
        upper = torch.where(go & neg & (r > 0.0), p, upper)
        lower = torch.where(go & neg & ~(r > 0.0), p, lower)
        new = p - r / dr
        bad = ~torch.isfinite(new) | (new <= lower) | (new >= upper)
        new = torch.where(bad, 0.5 * (lower + upper), new)
        p = torch.where(go, new, p)
        r, dr = residual(p)
    e = tau + D + p
    v2 = S2 / (e * e)
    ok = ok & (r.abs() < tol) & (v2 < cap)
    rho = D * torch.sqrt(torch.clamp(1.0 - v2, min=0.0))
    return (rho, p, [m / e for m in mom]), ok


def _atmosphere(o, rho, p, factor):
    return (rho <= factor * o.rho_floor) & (p <= factor * o.pressure_floor)


def _fluxes(pr, U, d, lapse, shift):
    tv = lapse * pr[2][d] - shift[d]
    ap = lapse * pr[1]
    f = [U[0] * tv] + [U[1 + j] * tv for j in range(3)] + [
        U[4] * tv + ap * pr[2][d]]
    f[1 + d] = f[1 + d] + ap
    return f


def _speeds(o, pr, gLL, gUU, lapse, shift, d):
    rho, p, v, eps = pr
    v2 = _dot(_lower(gLL, v), v)
    cs2 = o.adiabatic_index * p / (rho * (1.0 + eps + p / rho))
    den = 1.0 - v2 * cs2
    rad = (1.0 - v2) * (gUU[_SYM[d][d]] * den - v[d] * v[d] * (1.0 - cs2))
    root = torch.sqrt(cs2) * torch.sqrt(torch.clamp(rad, min=0.0))
    base = v[d] * (1.0 - cs2)
    return (lapse * ((base - root) / den) - shift[d],
            lapse * ((base + root) / den) - shift[d])


def _minmod(a, b):
    m = torch.where(a > 0.0, torch.minimum(a, b), torch.maximum(a, b))
    return torch.where(a * b <= 0.0, torch.zeros_like(m), m)


def _slope(a, b, c, theta):
    return _minmod(theta * (b - a),
                   _minmod(0.5 * (c - a), theta * (c - b)))


def _face_fluxes(o, q, geo, d):
    """HLLE fluxes of the n + 1 faces of the interior along direction d."""
    dim = 2 - d
    g = 2
    n = [m - 2 * g for m in q[0].shape]

    def at(f, first):
        for a in range(3):
            f = f.narrow(a, first, n[a] + 1) if a == dim else \
                f.narrow(a, g, n[a])
        return f

    def face(f):
        return 0.5 * (at(f, g - 1) + at(f, g))

    gLL, gUU = [face(f) for f in geo.gLL], [face(f) for f in geo.gUU]
    lapse, shift = face(geo.lapse), [face(f) for f in geo.shift]
    left, right = [], []
    for f in q:
        c = [at(f, g - 2 + m) for m in range(4)]
        left.append(c[1] + 0.5 * _slope(c[0], c[1], c[2], o.limiter_theta))
        right.append(c[2] - 0.5 * _slope(c[1], c[2], c[3], o.limiter_theta))
    side = []
    for s in (left, right):
        pr = _floors(o, s[0], s[1], s[2:], gLL)
        U = _p2c(pr, gLL)
        side.append((U, _fluxes(pr, U, d, lapse, shift),
                     _speeds(o, pr, gLL, gUU, lapse, shift, d)))
    (UL, FL, sL), (UR, FR, sR) = side
    lo = torch.clamp(torch.minimum(sL[0], sR[0]), max=0.0)
    hi = torch.clamp(torch.maximum(sL[1], sR[1]), min=0.0)
    out = []
    for c in range(5):
        f = (hi * FL[c] - lo * FR[c] + lo * hi * (UR[c] - UL[c])) / (hi - lo)
        out.append(torch.where(lo >= 0.0, FL[c],
                               torch.where(hi <= 0.0, FR[c], f)))
    return out, gLL


def _static_sources(pr, U, geo):
    rho, p, v, eps = pr
    W2 = 1.0 / (1.0 - _dot(_lower(geo.gLL, v), v))
    rhw = rho * (1.0 + eps + p / rho) * W2
    st = [rhw * v[i] * v[j] + p * geo.gUU[q]
          for q, (i, j) in enumerate(_PAIR)]
    mU = _lower(geo.gUU, U[1:4])
    F = [_fluxes(pr, U, d, geo.lapse, geo.shift) for d in range(3)]
    vol = [-_dot([F[d][c] for d in range(3)], geo.dlnsqrtg)
           for c in range(5)]
    src = [vol[0], None, None, None,
           vol[4] - _dot(mU, geo.dlapse) + geo.lapse * _trace(st, geo.K)]
    for m in range(3):
        src[1 + m] = (vol[1 + m] - (U[0] + U[4]) * geo.dlapse[m]
                      + 0.5 * geo.lapse * _trace(st, geo.dgam[m])
                      + _dot(U[1:4], geo.dshift[m]))
    return src


def _inner(f):
    return f[..., 2:-2, 2:-2, 2:-2]


class _Scheme:
    """The scheme on one box that covers its domain, or (lo) on a patch whose
    ghosts lie inside it."""

    def __init__(self, p, state, inv, lo=None):
        self.o, self.inv = p, inv
        self.shape = state.shape[1:]
        self.glo = [(lo[d] if lo else 0) - 2 for d in range(3)]
        self.patch = lo is not None
        self.held = (None, None)
        self.mdot = None
        # excised cells keep the primitives the state holds
        self.frozen = [state[c] for c in (5, 7, 8, 9, 10)]
        self.src = []
        for n in self.shape:
            i = torch.arange(n, device=state.device)
            self.src.append(torch.clamp(i, 2, n - 3))
        self.ghost = torch.ones(self.shape, dtype=torch.bool,
                                device=state.device)
        _inner(self.ghost)[...] = False
        if self.patch:
            self.ghost[...] = False

    def geometry(self, t):
        if self.o.background == 0:
            t = 0.0
        if self.held[0] != t:
            self.held = (None, None)
            self.held = (t, _Geometry(self.o, self.glo, self.shape, t))
        return self.held[1]

    def outflow(self, f):
        z, y, x = self.src
        return f[z][:, y][:, :, x]

    def fill(self, U, geo):
        """The outflow ghosts: the edge cell's primitives, floored and made
        conserved with the ghost's own metric."""
        if self.patch:
            return U
        (rho, p, v), _ = _con2prim(self.o, U, geo.gUU)
        pr = _floors(self.o, self.outflow(rho), self.outflow(p),
                     [self.outflow(q) for q in v], geo.gLL)
        new = _p2c(pr, geo.gLL)
        return [torch.where(self.ghost, a, b) for a, b in zip(new, U)]

    def sources(self, q, U, geo):
        pr = _floors(self.o, q[0], q[1], q[2:], geo.gLL)
        out = [torch.zeros_like(U[0]) for _ in range(5)]
        if self.o.use_static_metric_sources:
            s = _static_sources(pr, U, geo)
            air = _atmosphere(self.o, pr[0], pr[1], max(
                1.0, self.o.metric_source_atmosphere_factor))
            out = [torch.where(air, z, f) for z, f in zip(out, s)]
        if geo.volume_rate is not None:
            out = [f - u * geo.volume_rate for f, u in zip(out, U)]
        return out

    def rhs(self, U, t):
        geo = self.geometry(t)
        U = self.fill(U, geo)
        (rho, p, v), _ = _con2prim(self.o, U, geo.gUU)
        q = [rho, p] + v
        if self.o.excision_radius > 0.0:
            hole = geo.excised & ~self.ghost
            q = [torch.where(hole, f, a) for f, a in zip(self.frozen, q)]
        out = [_inner(f) for f in self.sources(q, U, geo)]
        mdot = 0.0
        for d in range(3):
            F, gLL = _face_fluxes(self.o, q, geo, d)
            dim, n = 2 - d, self.shape[2 - d] - 4
            if self.o.accretion_radius > 0.0:
                mdot = mdot + self.face_mdot(F[0], gLL, geo.inside, d)
            out = [r - self.inv[d] * (f.narrow(dim, 1, n)
                                      - f.narrow(dim, 0, n))
                   for r, f in zip(out, F)]
            del F, gLL
        if self.o.excision_radius > 0.0:
            out = [torch.where(_inner(geo.excised), 0.0, r) for r in out]
        self.mdot = mdot
        return out

    def face_mdot(self, FD, gLL, inside, d):
        n = [m - 4 for m in self.shape]

        def at(first):
            f = inside
            for a in range(3):
                f = f.narrow(a, first, n[a] + 1) if a == 2 - d else \
                    f.narrow(a, 2, n[a])
            return f
        left, right = at(1).double(), at(2).double()
        return ((right - left) * torch.sqrt(_det(gLL)) * FD).sum() \
            * self.o.dx ** 2

    def recover(self, U, t):
        """The recovery after an update: floors, and the atmosphere where it
        fails.  Returns the conserved state and the primitives."""
        geo, o = self.geometry(t), self.o
        (rho, p, v), ok = _con2prim(o, U, geo.gUU)
        f = _floors(o, rho, p, v, geo.gLL)
        same = (f[0] == rho) & (f[1] == p)
        for a, b in zip(f[2], v):
            same = same & (a == b)
        zero = torch.zeros_like(rho)
        rho = torch.where(ok, f[0], zero + o.rho_floor)
        p = torch.where(ok, f[1], zero + o.pressure_floor)
        v = [torch.where(ok, a, zero) for a in f[2]]
        pr = (rho, p, v, _eps(o, rho, p))
        new = _p2c(pr, geo.gLL)
        keep = ok & same
        return [torch.where(keep, a, b) for a, b in zip(U, new)], pr

    def max_inverse_dt(self, U, t):
        geo, o = self.geometry(t), self.o
        (rho, p, v), _ = _con2prim(o, U, geo.gUU)
        pr = _floors(o, rho, p, v, geo.gLL)
        cell = 0.0
        for d in range(3):
            lo, hi = _speeds(o, pr, geo.gLL, geo.gUU, geo.lapse, geo.shift, d)
            cell = cell + torch.maximum(lo.abs(), hi.abs()) * self.inv[d]
        air = _atmosphere(o, pr[0], pr[1], 1.0 + 1e-12)
        if o.excision_radius > 0.0:
            air = air | geo.excised
        return float(_inner(torch.where(air, 0.0, cell)).max())

    def add(self, U, k, dt):
        out = []
        for u, f in zip(U, k):
            u = u.clone()
            _inner(u).add_(f, alpha=dt)
            out.append(u)
        return out

    def state(self, U, pr, old):
        """The 11 components, those of excised cells unchanged."""
        s = torch.stack(list(U) + [pr[0], pr[3], pr[1]] + list(pr[2]))
        if self.o.excision_radius > 0.0:
            s = torch.where(self.geometry(0.0).excised, old, s)
        return s

    def rk4(self, s, t, dt):
        """One step; the accretion integral of its stages is added up."""
        U0 = [s[c] for c in range(5)]
        k1 = self.rhs(U0, t)
        J = self.mdot
        U, _ = self.recover(self.add(U0, k1, 0.5 * dt), t + 0.5 * dt)
        k2 = self.rhs(U, t + 0.5 * dt)
        J = J + 2.0 * self.mdot
        acc = [a + 2.0 * b for a, b in zip(k1, k2)]
        U, _ = self.recover(self.add(U0, k2, 0.5 * dt), t + 0.5 * dt)
        k3 = self.rhs(U, t + 0.5 * dt)
        J = J + 2.0 * self.mdot
        acc = [a + 2.0 * b for a, b in zip(acc, k3)]
        U, _ = self.recover(self.add(U0, k3, dt), t + dt)
        k4 = self.rhs(U, t + dt)
        J = J + self.mdot
        acc = [a + b for a, b in zip(acc, k4)]
        U, pr = self.recover(self.add(U0, acc, dt / 6.0), t + dt)
        self.J = dt / 6.0 * J
        return self.state(U, pr, s)

    def ssprk2(self, s, t, dt, extra=None):
        """`extra(state, rhs, time)` adds to each right-hand side; `decay`
        multiplies the combined state."""
        U0 = [s[c] for c in range(5)]
        k = self.rhs(U0, t)
        if extra:
            k = extra(s, k, t)
        U1, pr = self.recover(self.add(U0, k, dt), t + dt)
        s1 = self.state(U1, pr, s)
        U1 = [s1[c] for c in range(5)]
        k = self.rhs(U1, t + dt)
        if extra:
            k = extra(s1, k, t + dt)
        return self.add([0.5 * (a + b) for a, b in zip(U0, U1)], k, 0.5 * dt)


class _GridMetric:
    """Geometry from the grid's CCZ4 variables."""

    def __init__(self, p, s, inv):
        chi, h = s[0], [s[1 + q] for q in range(6)]
        self.gLL = [f / chi for f in h]
        self.gUU = [chi * f for f in _inverse(h)]
        self.K = [s[8 + q] / chi + self.gLL[q] * s[7] / 3.0 for q in range(6)]
        self.lapse = s[18]
        self.shift = [s[19], s[20], s[21]]
        self.volume_rate = None
        air = _atmosphere(p, s[30], s[32],
                          max(1.0, p.metric_source_atmosphere_factor))
        lnd = 0.5 * torch.log(_det(self.gLL))
        self.dgam, self.dshift, self.dlapse, self.dlnsqrtg = [], [], [], []
        for d in range(3):
            dim = 2 - d
            lo_air, hi_air = air.roll(1, dim), air.roll(-1, dim)

            def diff(f, dim=dim, d=d, lo_air=lo_air, hi_air=hi_air):
                lo = torch.where(lo_air, f, f.roll(1, dim))
                hi = torch.where(hi_air, f, f.roll(-1, dim))
                diff = inv[d] * (hi - lo)
                diff = torch.where(lo_air | hi_air, diff, 0.5 * diff)
                return torch.where(lo_air & hi_air, 0.0, diff)
            self.dgam.append([diff(f) for f in self.gLL])
            self.dshift.append([diff(f) for f in self.shift])
            self.dlapse.append(diff(self.lapse))
            self.dlnsqrtg.append(diff(lnd))


class _GridScheme(_Scheme):
    """The scheme on a metric that the grid holds."""

    def __init__(self, p, state, inv):
        super().__init__(p, state[25:], inv)
        self.full = state
        for c in list(range(7)) + list(range(18, 22)):
            state[c] = self.outflow(state[c])

    def hold(self, s11):
        """The state whose stored primitives pick the source stencils."""
        full = self.full.clone()
        full[25:] = s11
        self.metric = _GridMetric(self.o, full, self.inv)

    def geometry(self, t):
        return self.metric

    def fill(self, U, geo):
        return [torch.where(self.ghost, self.outflow(u), u) for u in U]

    def step(self, s, dt):
        self.hold(s)
        U0 = [s[c] for c in range(5)]
        k = self.rhs(U0, 0.0)
        U0 = self.fill(U0, None)
        U1, pr = self.recover(self.add(U0, k, dt), 0.0)
        s1 = self.state(U1, pr, s)
        # ghosts keep the primitives that the state came with
        s1 = torch.where(self.ghost, torch.cat([s1[:5], s[5:]]), s1)
        self.hold(s1)
        U1 = [s1[c] for c in range(5)]
        k = self.rhs(U1, 0.0)
        U, pr = self.recover(self.add([0.5 * (a + b) for a, b in
                                       zip(U0, U1)], k, 0.5 * dt), 0.0)
        return self.state(U, pr, s)


class _Driver:
    """The disk driver's viscous stress and point-mass sinks."""

    def __init__(self, p, cfg, scheme):
        self.o, self.cfg, self.sch = p, cfg, scheme
        self.pos = scheme.geometry(0.0).pos

    def _r2(self, t, eps):
        out = []
        for pos, _ in _orbit(self.o, t)[0]:
            out.append(eps + sum((self.pos[d] - pos[d]) ** 2
                                 for d in range(3)))
        return out

    def viscous(self, s, rhs, t):
        o, c = self.o, self.cfg
        masses = (o.pn_mass_1, o.pn_mass_2)
        om2 = sum(m * r2 ** -1.5 for m, r2 in zip(masses, self._r2(t, 1e-10)))
        rho, p = _inner(s[5]), _inner(s[7])
        cs2 = o.adiabatic_index * p / torch.clamp(rho, min=c.rho_floor)
        mu = rho * c.alpha_viscosity * cs2 / torch.sqrt(
            torch.clamp(_inner(om2), min=1e-300))
        mu = torch.where(rho <= 10.0 * o.rho_floor, 0.0, mu)
        v = [_inner(s[8]), _inner(s[9])]
        grad = [[self._diff(v[a], b, o.dx, True) for b in range(2)]
                for a in range(2)]
        div = grad[0][0] + grad[1][1]
        out = list(rhs)
        for d in range(2):
            tau = [mu * (grad[d][a] + grad[a][d]
                         + (c.viscosity_beta - 2.0 / 3.0) * div * (a == d))
                   for a in range(2)]
            f = {1: -tau[0], 2: -tau[1], 4: -tau[0] * v[0] - tau[1] * v[1]}
            for comp, flux in f.items():
                out[comp] = out[comp] - self._diff(flux, d, o.dx, False)
        return out

    @staticmethod
    def _diff(f, d, dx, one_sided):
        """Central difference along d, clamped to the domain at its ends
        (divided by the cells it spans when one_sided)."""
        dim = 2 - d
        n = f.shape[dim]
        i = torch.arange(n, device=f.device)
        lo, hi = torch.clamp(i - 1, min=0), torch.clamp(i + 1, max=n - 1)
        span = (hi - lo).double() if one_sided else torch.full_like(
            i, 2, dtype=torch.float64)
        shape = [1, 1, 1]
        shape[dim] = n
        return (f.index_select(dim, hi) - f.index_select(dim, lo)) / (
            torch.clamp(span, min=1.0) * dx).reshape(shape)

    def decay(self, U, t, dt):
        rate = 0.0
        for m, r2 in zip((self.o.pn_mass_1, self.o.pn_mass_2),
                         self._r2(t, 0.0)):
            size = self.cfg.sink_size * m
            rate = rate + self.cfg.sink_rate * torch.exp(
                -(r2 / size ** 2) ** (0.5 * self.cfg.sink_shape))
        f = torch.where(U[0] > 0.0, torch.exp(-rate * dt), 1.0)
        return [torch.where(self.sch.ghost, u, u * f) for u in U]


def _exact_steps(op, state, inv, steps):
    sch = _Scheme(op.params, state, inv)
    mi = sch.max_inverse_dt([state[c] for c in range(5)], 0.0)
    t, s = 0.0, state
    for _ in range(steps):
        dt = CFL / mi
        s = sch.rk4(s, t, dt)
        t += dt
        mi = sch.max_inverse_dt([s[c] for c in range(5)], t)
    return sch, s, mi


def exact(case, seed):
    s = prepare(case, seed)
    work = case["work"]
    if work == "ensemble":
        out = []
        for op, lv in s["members"]:
            inv = [1.0 / op.dx] * 3
            out.append(_inner(_exact_steps(op, lv.state, inv,
                                           case["steps"])[1]))
        return out
    op, p = s["op"], s["op"].params
    if work == "adjoint":
        state = s["adj"].initial_state().state
        sch = _Scheme(p, state, [1.0 / op.dx] * 3)
        J = 0.0
        for _ in range(case["steps"]):
            state = sch.rk4(state, 0.0, s["dt"])
            J += float(sch.J)
        return dict(J=J, grad=None)
    inv = s["inv"]
    if work == "rhs":
        sch = _Scheme(p, s["lv"].state, inv,
                      s["lv"].lo if case["flow"] == "torus" else None)
        return torch.stack(sch.rhs([s["lv"].state[c] for c in range(5)], 0.0))
    if work == "ccz4":
        sch = _GridScheme(s["cop"].params, s["lv"].state, inv)
        state = s["lv"].state[25:]
        sch.hold(state)
        dt = CFL / sch.max_inverse_dt([state[c] for c in range(5)], 0.0)
        return _inner(sch.step(state, dt))
    if work == "host":
        state = s["host"].cuda()
        return _inner(_exact_steps(op, state, inv, 1)[1]).cpu()
    if work == "rk4":
        sch, state, mi = _exact_steps(op, s["lv"].state, inv, case["steps"])
        out = dict(state=_inner(state), next_max_inverse_dt=mi)
        if case["flow"] == "michel":
            out["mdot"] = float(sch.mdot)
        return out
    if work == "level":
        lv = _flow(case, seed)[1]
        state = lv.state
        sch = _Scheme(p, state, inv)
        dt = CFL / sch.max_inverse_dt([state[c] for c in range(5)], 0.0)
        U, pr = sch.recover(sch.ssprk2(state, 0.0, dt), dt)
        new = sch.state(U, pr, state)
        return [new[:, b.lo[2] + 2:b.hi[2] + 3, b.lo[1] + 2:b.hi[1] + 3,
                    b.lo[0] + 2:b.hi[0] + 3] for b in s["boxes"]]
    state = s["lv"].state  # the disk driver's step
    sch = _Scheme(p, state, inv)
    drv = _Driver(p, s["cfg"], sch)
    dt = CFL / sch.max_inverse_dt([state[c] for c in range(5)], 0.0)
    U = sch.ssprk2(state, 0.0, dt, drv.viscous)
    U, pr = sch.recover(drv.decay(U, 0.5 * dt, dt), dt)
    return _inner(sch.state(U, pr, state))
