"""What a user of this package has it do, as cases that can be timed and checked.

Every case goes through the public classes: ``DGSEMOperator`` (one solve: ``Mult``
for the right-hand side, ``Step`` for Runge-Kutta steps) or ``Batch`` (many solves
advanced together).  Meshes are axis-aligned boxes, so that ``exact`` can evaluate
the same discretisation with plain tensor operations in 64 bits: the split-form
DGSEM of entropy-conservative two-point fluxes on Gauss-Lobatto nodes, the BR1
lifting, the no-slip walls, the subcell blending and both Runge-Kutta schemes.

States are laid out as ``u[f, element, node]`` flattened, fields (rho, rho v, E),
elements and nodes lexicographic with x fastest.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from prandtl_b200.batch import Batch
from prandtl_b200.mesh import periodic_box
from prandtl_b200.operator import DGSEMOperator

GAMMA = 1.4
PR = 0.71
TWO_PI = 2.0 * math.pi
R_GAS = 1.0   # of the channel flow, so that a temperature is p / rho
# gas constant apart, these are the operator's own defaults
ALPHA_MAX, ALPHA_MIN = 0.5, 0.001

# elements per direction and order of the solves of a serving queue: 2D Euler
# vortices (n up to 128, N 3..4) and 3D Taylor-Green vortices (n up to 24, N 2..3)
SERVING_2D, SERVING_3D = (16, 128), (8, 24)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one right-hand side of the 2D isentropic vortex, 32^2 elements: the smallest
        # solve that is run in earnest; launches and the host count
        dict(name="vortex32_rhs", kind="vortex", dim=2, n=32, order=3, call="mult"),
        # ten steps of a larger 2D vortex at an odd size: the run loop of a small solve
        dict(name="vortex101_steps", kind="vortex", dim=2, n=101, order=4, call="step", scheme="LSRK45", steps=10),
        # shock-capturing Kelvin-Helmholtz instability at 256^2 elements, one SSP-RK3 step
        dict(name="kh256_blended_step", kind="kh", dim=2, n=256, order=3, call="step", scheme="RK3SSP", steps=1),
        # viscous channel between a fixed adiabatic and a moving isothermal wall
        dict(name="channel_walls_step", kind="channel", dim=2, n=120, order=4, call="step", scheme="RK3SSP", steps=1),
        # the 32^3 Taylor-Green vortex in FP64: one right-hand side, on device arrays
        dict(name="tgv32_rhs", kind="tgv", dim=3, n=32, order=3, call="mult", quirks="fixed"),
        # the same call on host arrays, as a CPU time integrator makes it
        dict(name="tgv24_rhs_host", kind="tgv", dim=3, n=24, order=3, call="host", quirks="fixed"),
        # the operator's default mode, which reproduces the reference's viscous terms
        dict(name="tgv20_rhs_reference", kind="tgv", dim=3, n=20, order=3, call="mult", quirks="reference"),
        # 3D Navier-Stokes steps in FP64 at a higher order and an odd size
        dict(name="tgv15_step_N4", kind="tgv", dim=3, n=15, order=4, call="step", scheme="LSRK45", steps=1,
             quirks="fixed"),
        # inviscid 3D flow in FP64
        dict(name="euler24_rhs", kind="euler", dim=3, n=24, order=3, call="mult"),
        # one solve in the FP32-bulk form at the highest order
        dict(name="tgv16_step_fp32_N5", kind="tgv", dim=3, n=16, order=5, call="step", scheme="LSRK45", steps=1,
             quirks="fixed", precision="fp32"),
        # a serving queue's mix of small 2D and 3D solves, untuned, monitored after every step
        dict(name="serving_mix_fp32", kind="serving", members=17, count=16, call="batch", steps=1),
        # an ensemble of uneven Taylor-Green vortices (4..16 elements per direction,
        # N 2..5): the throughput workload
        dict(name="ensemble96_fp32", kind="ensemble", members=5, count=96, call="batch", steps=1, tune=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vortex", "kh", "channel", "tgv", "tgv", "tgv", "euler", "serving", "ensemble", "ensemble"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randrange(1, 1 << 20), count=_log_int(rng, 3, 64), call="batch",
                    steps=rng.choice([1, 1, 2]), tune=rng.random() < 0.5)
    if kind == "serving":
        return dict(kind=kind, members=rng.randrange(1, 1 << 20), count=_log_int(rng, 2, 32), call="batch",
                    steps=rng.choice([1, 1, 2]))
    case = dict(kind=kind, dim=2 if kind in ("vortex", "kh", "channel") else 3)
    case["order"] = rng.choice([1, 2, 3, 3, 4, 5]) if kind != "kh" else rng.choice([2, 3, 3, 4])
    # nodes per direction spread over the range, whatever the order
    nodes = _log_int(rng, 48, 1200) if case["dim"] == 2 else _log_int(rng, 16, 120)
    case["n"] = max(3, nodes // (case["order"] + 1))
    if kind == "tgv":
        case["quirks"] = rng.choice(["fixed", "fixed", "reference"])
        # the FP32-bulk form is for taking steps
        case["precision"] = rng.choice(["fp64", "fp32"]) if case["quirks"] == "fixed" else "fp64"
    # the reference's own viscous terms are evaluated, not marched (they are not entropy stable in 3D)
    if case.get("quirks") == "reference" or case.get("precision") != "fp32" and rng.random() < 0.5:
        case["call"] = "host" if rng.random() < 0.2 else "mult"
    else:
        steps = [1, 2] if case.get("precision") == "fp32" else [1, 2, 9]
        case.update(call="step", scheme=rng.choice(["LSRK45", "RK3SSP"]), steps=rng.choice(steps))
    return case


# ------------------------------------------------------- meshes and parameters
def _box(kind, dim):
    """(lower corner, upper corner) of the domain."""
    if kind == "vortex":
        return (0.0,) * dim, (10.0,) * dim
    if kind == "kh":
        return (-1.0,) * dim, (1.0,) * dim
    if kind == "channel":
        return (0.0, 0.0), (TWO_PI, 2.0)
    return (0.0,) * dim, (TWO_PI,) * dim


@functools.lru_cache(maxsize=None)
def _mesh(kind, dim, n, order):
    lo, hi = _box(kind, dim)
    bcs = [None, None, 0, 1] if kind == "channel" else None
    return periodic_box(dim, _cells(kind, dim, n), order, lo, hi, bcs=bcs)


def _cells(kind, dim, n):
    return (n, max(2, n // 2)) if kind == "channel" else (n,) * dim


def _flow(case, seed):
    """Random parameters of one solve's initial state and its gas, from the seed."""
    r = random.Random("%s %s" % (seed, sorted((k, v) for k, v in case.items() if k in ("kind", "n", "order", "index"))))
    flow = dict(kind=case["kind"], shift=[r.uniform(0.0, 1.0) for _ in range(3)], tilt=r.uniform(0.8, 1.2),
                mach=math.exp(r.uniform(math.log(0.05), math.log(0.3))),
                re=math.exp(r.uniform(math.log(100.0), math.log(3200.0))))
    if case["kind"] == "channel":
        flow["mach"] = r.uniform(0.2, 0.4)
    return flow


def _physics(case, flow):
    """The operator's keyword arguments."""
    kind = case["kind"]
    if kind == "kh":
        return dict(blending=True, alpha_max=ALPHA_MAX)
    if kind == "tgv":
        return dict(parabolic=True, mu=1.0 / flow["re"], Pr=PR, quirks=case.get("quirks", "fixed"))
    if kind == "channel":
        return dict(parabolic=True, mu=1.0 / flow["re"], Pr=PR, quirks="fixed", R_gas=R_GAS, bcs=_walls(flow))
    return dict(quirks="fixed")


def _walls(flow):
    p0 = 1.0 / (GAMMA * flow["mach"] ** 2)
    return [("noslip_adiabatic", dict(wall_vel=(0.0, 0.0), heat_flux=0.0)),
            ("noslip_isothermal", dict(wall_vel=(1.0, 0.0), wall_T=1.02 * p0 / R_GAS))]


def _dt(kind, dim, n, order, flow):
    """The ensembles' own step: CFL 0.1, dt = 0.1 h / (lambda (N+1)^2)."""
    lo, hi = _box(kind, dim)
    h = min((b - a) / c for a, b, c in zip(lo, hi, _cells(kind, dim, n)))
    speed = {"vortex": 4.0, "kh": 4.0}.get(kind, 1.5 + 1.0 / flow["mach"])
    return 0.1 * h / (speed * (order + 1) ** 2)


def _members(case):
    """The solves of a batch: shapes from the case, kinds as single cases."""
    r = random.Random(case["members"])
    out = []
    for k in range(case["count"]):
        if case["kind"] == "ensemble":
            m = dict(kind="tgv", dim=3, n=r.randint(4, 16), order=r.randint(2, 5))
        elif r.random() < 0.5:
            m = dict(kind="vortex", dim=2, n=r.randint(*SERVING_2D), order=r.randint(3, 4))
        else:
            m = dict(kind="tgv", dim=3, n=r.randint(*SERVING_3D), order=r.randint(2, 3))
        out.append(dict(m, index=k))
    return out


# -------------------------------------------------------------- initial states
@functools.lru_cache(maxsize=None)
def _rule(order):
    """Gauss-Lobatto nodes and weights on [0, 1], D, and the inverse Legendre Vandermonde matrix."""
    N = order
    leg = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(leg.deriv().roots().real), [1.0]])
    for _ in range(3):   # polish the interior roots of P'_N
        x[1:-1] -= leg.deriv()(x[1:-1]) / leg.deriv(2)(x[1:-1])
    w = 2.0 / (N * (N + 1) * leg(x) ** 2)
    V = np.polynomial.legendre.legvander(x, N)
    D = np.stack([np.polynomial.legendre.Legendre.basis(k).deriv()(x) if k else 0 * x for k in range(N + 1)], 1) @ np.linalg.inv(V)
    D -= np.diag(D.sum(axis=1))
    return 0.5 * (x + 1.0), 0.5 * w, 2.0 * D, np.linalg.inv(V)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _coords(kind, dim, n, order):
    """Node coordinates, each shaped to broadcast over [cells z, y, x, nodes k, j, i]."""
    x1 = torch.from_numpy(_rule(order)[0]).to(_device())
    lo, hi = _box(kind, dim)
    cells = _cells(kind, dim, n)
    out = []
    for d in range(dim):
        c = torch.arange(cells[d], dtype=torch.float64, device=x1.device)
        x = lo[d] + (c[:, None] + x1[None, :]) * ((hi[d] - lo[d]) / cells[d])
        shape = [1] * (2 * dim)
        shape[dim - 1 - d], shape[2 * dim - 1 - d] = cells[d], order + 1
        out.append(x.reshape(shape))
    return out


def _initial(case, flow):
    """The flattened state of one solve, made on the device."""
    kind, dim = case["kind"], case["dim"]
    X = _coords(kind, dim, case["n"], case["order"])
    s = flow["shift"]
    g1 = GAMMA - 1.0
    if kind == "vortex":   # isentropic vortex in a uniform stream
        x, y = X[0] - (4.0 + 2.0 * s[0]), X[1] - (4.0 + 2.0 * s[1])
        r2, eps = x * x + y * y, 4.0 + s[2]
        f = torch.exp(0.5 * (1.0 - r2)) * (eps / TWO_PI)
        T = 1.0 - g1 / (2.0 * GAMMA) * f * f
        rho = T ** (1.0 / g1)
        vel, p = [1.0 - f * y, 1.0 + f * x], rho * T
    elif kind == "kh":   # smoothed double shear layer with a transverse perturbation
        x, y = X
        B = torch.tanh(15.0 * y + 7.5) - torch.tanh(15.0 * y - 7.5) + 0.0 * x
        rho = 0.5 + 0.75 * B
        vel = [0.5 * (B - 1.0), 0.1 * torch.sin(TWO_PI * (x + s[0])) + 0.02 * torch.sin(2 * TWO_PI * (x + s[1])) + 0.0 * y]
        p = torch.ones_like(rho)
    elif kind == "channel":   # shear flow between the walls with a decaying wave on it
        x, y = X
        p0 = 1.0 / (GAMMA * flow["mach"] ** 2)
        wave = torch.sin(0.5 * math.pi * y) ** 2
        vel = [0.5 * y + 0.1 * wave * torch.sin(x + TWO_PI * s[0]), 0.05 * wave * torch.cos(2 * x + TWO_PI * s[1])]
        p = p0 * (1.0 + 0.01 * torch.cos(x + TWO_PI * s[2]) * torch.cos(math.pi * y))
        rho = 1.0 + 0.02 * torch.sin(x + TWO_PI * s[0]) * torch.cos(0.5 * math.pi * y)
    else:   # Taylor-Green vortex, shifted and slightly stretched in amplitude
        x, y, z = [c + TWO_PI * a for c, a in zip(X, s)]
        a = flow["tilt"]
        p0 = 1.0 / (GAMMA * flow["mach"] ** 2)
        vel = [a * torch.sin(x) * torch.cos(y) * torch.cos(z), -a * torch.cos(x) * torch.sin(y) * torch.cos(z), None]
        p = p0 + (a * a / 16.0) * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)
        rho = p / p0
        vel[2] = torch.zeros_like(rho)
    E = p / g1 + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho + 0.0 * E] + [rho * v + 0.0 * E for v in vel] + [E]).reshape(-1).contiguous()


# ------------------------------------------------------------- prepare and run
def prepare(case, seed):
    if case["call"] == "batch":
        return _prepare_batch(case, seed)
    flow = _flow(case, seed)
    u = _initial(case, flow)
    mesh = _mesh(case["kind"], case["dim"], case["n"], case["order"])
    op = DGSEMOperator(mesh, precision=case.get("precision", "fp64"), **_physics(case, flow))
    if u.is_cuda:
        op.set_stream(torch.cuda.current_stream().cuda_stream)
    state = dict(case=case, op=op)
    if case["call"] == "host":
        u = u.cpu().numpy()
        state.update(u=u, dudt=np.empty_like(u))
    else:
        state.update(u=u, dudt=torch.empty_like(u),
                     dt=_dt(case["kind"], case["dim"], case["n"], case["order"], flow))
    return state


def _prepare_batch(case, seed):
    solves, states = [], []
    for m in _members(case):
        flow = _flow(m, seed)
        phys = dict(_physics(m, flow), dt=_dt(m["kind"], m["dim"], m["n"], m["order"], flow), nsteps=10 ** 9)
        states.append(_initial(m, flow))
        solves.append((_mesh(m["kind"], m["dim"], m["n"], m["order"]), states[-1], phys))
    sizes = [u.numel() for u in states]
    # a solve holds three states, its gradients and its mesh tables: at most 3 + 3 states' worth and a fifth
    b = Batch("fp32", "LSRK45", arena_bytes=int(sum(8 * 6 * 1.2 * s + (1 << 20) for s in sizes)))
    torch.cuda.synchronize()
    ids = b.add_many(solves)
    b.sync()
    if case.get("tune"):
        b.tune()
    out = torch.empty(sum(sizes), dtype=torch.float64, device=states[0].device)
    return dict(case=case, batch=b, ids=ids, out=out, views=list(torch.split(out, sizes)))


def run(state):
    case = state["case"]
    if case["call"] == "batch":
        state["batch"].advance(case["steps"])
        state["batch"].read_many(state["ids"], state["views"])
        return state["out"]
    op = state["op"]
    if case["call"] == "step":
        return op.Step(state["u"], state["dt"], scheme=case["scheme"], nsteps=case["steps"])
    return op.Mult(state["u"], state["dudt"]), op.GetMaxCharSpeed()


# ------------------------------------------------------------------------ work
def _solve_work(case, evaluations):
    """(flops, state values) of so many right-hand sides of one solve (add, mul, div, sqrt, log count 1)."""
    dim, Np = case["dim"], case["order"] + 1
    nd, nf = Np ** dim, dim + 2
    E = math.prod(_cells(case["kind"], dim, case["n"]))
    viscous = case["kind"] in ("tgv", "channel")
    pairs, face_nodes = dim * nd * (Np - 1) // 2, dim * nd // Np   # every face is shared by two elements
    flops = pairs * (123 + 4 * nf) + face_nodes * (150 + 4 * nf) + nd * (20 + 6 * nf)
    if viscous:   # entropy variables, gradients and their lifting, viscous fluxes and their divergence
        flops += nd * (40 + 2 * dim * Np * nf + 2 * dim * dim * nf + dim * 30 + 60 + 2 * dim * Np * (nf - 1))
        flops += face_nodes * nf * (2 + 4 * dim)
    return evaluations * E * flops, E * nd * nf


def work(case):
    """Each state read once and each result written once: what no implementation of the call can do without."""
    stages = {"LSRK45": 5, "RK3SSP": 3}.get(case.get("scheme"), 1)
    if case["call"] == "batch":
        solves, evaluations = _members(case), 5 * case["steps"]
    else:
        solves, evaluations = [case], stages * case.get("steps", 1)
    done = [_solve_work(m, evaluations) for m in solves]
    return {"bytes": 16.0 * sum(v for _, v in done), "flops": float(sum(f for f, _ in done))}


# ------------------------------------------- the same discretisation, in 64 bits
def exact(case, seed):
    with torch.no_grad():
        if case["call"] == "batch":
            out = []
            for m in _members(case):
                flow = _flow(m, seed)
                out.append(_advance(m, flow, _initial(m, flow), "LSRK45", case["steps"]))
            return torch.cat(out)
        flow = _flow(case, seed)
        u = _initial(case, flow)
        if case["call"] == "step":
            return _advance(case, flow, u, case["scheme"], case["steps"])
        box = _Box(case, flow)
        U = box.shaped(u)
        q = _prim(U)
        lam = float((q["lam"]).max())
        dudt = box.rhs(U).reshape(-1)
        return (dudt.cpu().numpy() if case["call"] == "host" else dudt), lam


_LSRK_A = [0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
           -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0]
_LSRK_B = [1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
           1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
           2277821191437.0 / 14882151754819.0]


def _advance(case, flow, u, scheme, steps):
    box = _Box(case, flow)
    dt = _dt(case["kind"], case["dim"], case["n"], case["order"], flow)
    U = box.shaped(u)
    for _ in range(steps):
        if scheme == "LSRK45":
            dU = torch.zeros_like(U)
            for A, B in zip(_LSRK_A, _LSRK_B):
                dU = A * dU + dt * box.rhs(U)
                U = U + B * dU
        else:   # Shu-Osher
            y = U + dt * box.rhs(U)
            y = 0.75 * U + 0.25 * (y + dt * box.rhs(y))
            U = U / 3.0 + 2.0 / 3.0 * (y + dt * box.rhs(y))
    return U.reshape(-1)


def _prim(U):
    """Primitive variables of states U[f, ...]."""
    rho, E = U[0], U[-1]
    v = [m / rho for m in U[1:-1]]
    vsq = sum(c * c for c in v)
    p = (GAMMA - 1.0) * (E - 0.5 * rho * vsq)
    return dict(U=U, rho=rho, v=v, vsq=vsq, p=p, beta=0.5 * rho / p, lam=vsq.sqrt() + (GAMMA * p / rho).sqrt())


def _log_mean(x, y):
    f = (y - x) / (y + x)
    u = f * f
    series = (x + y) * 52.5 / (105.0 + u * (35.0 + u * (21.0 + 15.0 * u)))
    return torch.where(u < 1e-4, series, (y - x) / torch.log(y / x))


def _flux(a, b, d):
    """Chandrashekar's two-point flux in direction d, and what its dissipation needs."""
    rho_ln, beta_ln = _log_mean(a["rho"], b["rho"]), _log_mean(a["beta"], b["beta"])
    vm = [0.5 * (x + y) for x, y in zip(a["v"], b["v"])]
    p_hat = 0.5 * (a["rho"] + b["rho"]) / (a["beta"] + b["beta"])
    h = 0.5 / ((GAMMA - 1.0) * beta_ln) + p_hat / rho_ln - 0.25 * (a["vsq"] + b["vsq"]) + sum(c * c for c in vm)
    F0 = rho_ln * vm[d]
    F = torch.stack([F0] + [F0 * c + (p_hat if q == d else 0.0) for q, c in enumerate(vm)] + [F0 * h])
    return F, vm, beta_ln


def _face_flux(a, b, d, sign, aliased):
    """Surface flux along sign * e_d from a to b.  aliased: the reference's 3D energy dissipation."""
    F, vm, beta_ln = _flux(a, b, d)
    dim, g1 = len(vm), GAMMA - 1.0
    rho_mean, drho = 0.5 * (a["rho"] + b["rho"]), b["rho"] - a["rho"]
    diss = 0.5 * drho / (g1 * beta_ln) + 0.5 * rho_mean / g1 * (1.0 / b["beta"] - 1.0 / a["beta"])
    for q in range(dim):
        dv = b["v"][q] - a["v"][q]
        diss = diss + 0.5 * drho * a["v"][q] * b["v"][q]
        diss = diss + (rho_mean * dv + vm[q] if aliased and dim == 3 and q == 2 else rho_mean * dv * vm[q])
    jump = torch.cat([(b["U"] - a["U"])[:-1], diss[None]])
    return sign * F - 0.5 * torch.maximum(a["lam"], b["lam"]) * jump


def _at(q, pick):
    """The primitive variables at some of the nodes."""
    return {k: ([pick(c) for c in x] if k == "v" else pick(x)) for k, x in q.items()}


class _Box:
    """Right-hand side on an axis-aligned box, periodic but for the channel's walls in y."""

    def __init__(self, case, flow):
        self.dim, self.Np, self.kind = case["dim"], case["order"] + 1, case["kind"]
        self.cells = _cells(self.kind, self.dim, case["n"])
        lo, hi = _box(self.kind, self.dim)
        self.h = [(b - a) / c for a, b, c in zip(lo, hi, self.cells)]
        x, w, D, Vinv = _rule(case["order"])
        dev = _device()
        split = 2.0 * D
        split[0, 0] += 1.0 / w[0]
        split[-1, -1] -= 1.0 / w[-1]
        weak = D.copy()
        weak[0, 0] += 1.0 / w[0]
        weak[-1, -1] -= 1.0 / w[-1]
        self.w, self.w0 = torch.from_numpy(w).to(dev), float(w[0])
        self.D, self.split, self.weak, self.Vinv = (torch.from_numpy(np.ascontiguousarray(m)).to(dev) for m in (D, split, weak, Vinv))
        self.pairs = [torch.tensor(t, device=dev) for t in zip(*[(i, l) for i in range(self.Np) for l in range(i + 1, self.Np)])]
        phys = _physics(case, flow)
        self.viscous = bool(phys.get("parabolic"))
        self.mu = phys.get("mu", 0.0)
        self.reference = phys.get("quirks", "reference") == "reference"
        self.blending = bool(phys.get("blending"))
        self.walls = phys.get("bcs")

    def shaped(self, u):
        return u.reshape([self.dim + 2, *reversed(self.cells), *[self.Np] * self.dim])

    # directions as tensor axes
    def _line(self, d):
        return -1 - d

    def _cell(self, d):
        return -1 - d - self.dim

    def _along(self, M, x, d):
        """M applied along the lines of direction d."""
        return torch.movedim(torch.movedim(x, self._line(d), -1) @ M.T, -1, self._line(d))

    def _face_node(self, x, d, i):
        return x.select(self._line(d), i)

    def _next(self, x, d, by):
        """x, one cell further along d, of arrays that have lost the line axis of d."""
        return torch.roll(x, by, self._cell(d) + 1)

    def _last(self, x, d):
        """Mask of the wrap-around faces (those above the last cells) for arrays without d's line axis."""
        n = self.cells[d]
        shape = [1] * (2 * self.dim - 1)
        shape[self._cell(d) + 1] = n
        return (torch.arange(n, device=x.device) == n - 1).reshape(shape)

    def rhs(self, U):
        q = _prim(U)
        # reference mode only: the surface flux has its 3D energy dissipation written down as published there
        aliased = self.reference
        alpha = self._alpha(q) if self.blending else None
        out = torch.zeros_like(U)
        for d in range(self.dim):
            term = self._volume(q, d)
            if alpha is not None:
                term = (1.0 - alpha) * term + alpha * self._subcells(q, d, aliased)
            out += term / self.h[d]
        grads = self._gradients(q) if self.viscous else None
        if self.viscous:
            at = q
            if self.reference:   # volume viscous fluxes take the state of each element's last node
                last = (Ellipsis,) + (slice(self.Np - 1, self.Np),) * self.dim
                at = _at(q, lambda x: x[last])
            for d, F in enumerate(self._viscous(at, grads)):
                out += self._along(self.weak, F, d) / self.h[d]
        own = self._viscous(q, grads) if self.viscous else None
        traces = q
        if self.viscous and self.reference:   # the surface flux reads velocities in the momentum slots
            traces = _prim(torch.stack([U[0], *q["v"], U[-1]]))
        for d in range(self.dim):
            self._surface(out, q, traces, own[d] if own else None, d, aliased)
        return out

    def _volume(self, q, d):
        """-sum_l (2D + B)(i, l) F(i, l) along the lines of direction d."""
        ax, (ia, ib) = self._line(d), self.pairs
        F, _, _ = _flux(_at(q, lambda x: x.index_select(ax, ia)), _at(q, lambda x: x.index_select(ax, ib)), d)
        below = F
        if self.viscous and self.reference and self.dim == 3 and d == 2:
            # a node's lower partners contribute the y flux between the partner and its line's last node
            G, _, _ = _flux(q, _at(q, lambda x: x.narrow(-2, self.Np - 1, 1)), 1)
            G[..., self.Np - 1, :] = 0.0
            below = G.index_select(ax, ia) * (self.h[2] / self.h[1])
        shape = [1] * F.dim()
        shape[ax] = len(ia)
        out = torch.zeros_like(q["U"])
        out.index_add_(out.dim() + ax, ia, -F * self.split[ia, ib].reshape(shape))
        out.index_add_(out.dim() + ax, ib, -below * self.split[ib, ia].reshape(shape))
        return out

    def _subcells(self, q, d, aliased):
        """First-order finite volumes between the nodes of a line."""
        ax, Np = self._line(d), self.Np
        F = _face_flux(_at(q, lambda x: x.narrow(ax, 0, Np - 1)), _at(q, lambda x: x.narrow(ax, 1, Np - 1)), d, 1.0, aliased)
        out = torch.zeros_like(q["U"])
        out.narrow(ax, 0, Np - 1).sub_(F)
        out.narrow(ax, 1, Np - 1).add_(F)
        shape = [1] * out.dim()
        shape[ax] = Np
        return out / self.w.reshape(shape)

    def _alpha(self, q):
        """Blending factor from the decay of the Legendre modes of rho p."""
        m = q["rho"] * q["p"]
        for d in range(self.dim):
            m = self._along(self.Vinv, m, d)
        e = m * m
        axes = tuple(self._line(d) for d in range(self.dim))
        low = [e[(Ellipsis,) + (slice(0, k),) * self.dim].sum(axes, keepdim=True) for k in (self.Np, self.Np - 1, self.Np - 2)]
        eta = torch.maximum(1.0 - low[1] / low[0], 1.0 - low[2] / low[1])
        T = 0.5 * 10.0 ** (-1.8 * (self.Np - 1) ** 0.25)
        a = 1.0 / (1.0 + torch.exp(-9.21024 * (eta - T) / T))
        a = torch.where(a < ALPHA_MIN, torch.zeros_like(a), torch.where(a > 1.0 - ALPHA_MIN, torch.ones_like(a), a))
        return a.clamp(max=ALPHA_MAX)

    def _surface(self, out, q, traces, viscous, d, aliased):
        ax, Np, scale = self._line(d), self.Np, 1.0 / (self.w0 * self.h[d])
        hi = _at(traces, lambda x: self._face_node(x, d, Np - 1))
        lo = _at(traces, lambda x: self._next(self._face_node(x, d, 0), d, -1))
        f = _face_flux(hi, lo, d, 1.0, aliased)
        if aliased and self.dim == 3:   # there the flux depends on which element comes first: on wrap faces the upper one
            f = torch.where(self._last(f, d), -_face_flux(lo, hi, d, -1.0, aliased), f)
        if viscous is not None:
            f = f - 0.5 * (self._face_node(viscous, d, Np - 1) + self._next(self._face_node(viscous, d, 0), d, -1))
        above, below = f, self._next(f, d, 1)
        if self.walls and d == 1:
            above, below = above.clone(), below.clone()
            for side, node, cell in ((1, Np - 1, self.cells[1] - 1), (-1, 0, 0)):
                s = _at(q, lambda x: self._face_node(x, d, node).select(self._cell(d) + 1, cell))
                v = self._face_node(viscous, d, node).select(self._cell(d) + 1, cell)
                (above if side > 0 else below).select(self._cell(d) + 1, cell).copy_(self._wall_flux(s, v, side))
        out.select(ax, Np - 1).sub_(scale * above)
        out.select(ax, 0).add_(scale * below)

    def _wall_flux(self, s, viscous, side):
        """Flux along +y at a wall: the pressure of the wall's Riemann problem and the viscous flux."""
        g, g1 = GAMMA, GAMMA - 1.0
        rho, p, un = s["rho"], s["p"], side * s["v"][1]
        an = (g * p / rho).sqrt()
        shock = p + 0.25 * un * (g + 1.0) * rho * (un + (un * un + 8.0 / (g + 1.0) / rho * p * (g1 / (g + 1.0) + 1.0)).sqrt())
        fan = p * torch.clamp(1.0 + 0.5 * g1 * un / an, min=0.0001) ** (2.0 * g / g1)
        F = torch.zeros_like(viscous)
        F[2] = torch.where(un > 0.0, shock, fan)
        kind, data = self.walls[1 if side > 0 else 0]
        viscous = viscous.clone()
        if kind == "noslip_adiabatic":
            viscous[-1] = sum(V * viscous[1 + k] for k, V in enumerate(data["wall_vel"])) + side * data["heat_flux"]
        return F - viscous

    def _gradients(self, q):
        """BR1-lifted gradients of (rho, v, p) by way of the entropy variables."""
        g1 = GAMMA - 1.0
        rho, v, p = q["rho"], q["v"], q["p"]
        b = rho / p
        ent = torch.stack([(GAMMA - torch.log(p) + GAMMA * torch.log(rho)) / g1 - 0.5 * b * q["vsq"]] + [b * c for c in v] + [-b])
        grads = []
        for d in range(self.dim):
            g = self._along(self.D, ent, d) / self.h[d]
            hi = self._face_node(ent, d, self.Np - 1)
            half = 0.5 * (self._next(self._face_node(ent, d, 0), d, -1) - hi)
            above, below = half, self._next(half, d, 1)
            if self.walls and d == 1:
                above, below = above.clone(), below.clone()
                for side, node, cell in ((1, self.Np - 1, self.cells[1] - 1), (-1, 0, 0)):
                    e = self._face_node(ent, d, node).select(self._cell(d) + 1, cell)
                    kind, data = self.walls[1 if side > 0 else 0]
                    wb = -e[-1] if kind == "noslip_adiabatic" else torch.full_like(e[-1], 1.0 / (R_GAS * data["wall_T"]))
                    wall = torch.stack([e[0]] + [V * wb for V in data["wall_vel"]] + [-wb])
                    (above if side > 0 else below).select(self._cell(d) + 1, cell).copy_(side * (wall - e))
            g.select(self._line(d), self.Np - 1).add_(above / (self.w0 * self.h[d]))
            g.select(self._line(d), 0).add_(below / (self.w0 * self.h[d]))
            gv = [p / rho * (g[1 + k] + c * g[-1]) for k, c in enumerate(v)]
            # reference mode reads velocities where the momentum is meant
            acc = sum((c if self.reference else rho * c) * x for c, x in zip(v, gv))
            gr = rho * g[0] - g[-1] * (0.5 * rho * q["vsq"] - p / g1) + rho / p * acc
            grads.append([gr, *gv, p / rho * (gr + p * g[-1])])
        return grads

    def _viscous(self, q, grads):
        """Viscous flux of each direction: Stokes stress and Fourier heat flux."""
        dim, rho, v, p = self.dim, q["rho"], q["v"], q["p"]
        div = sum(grads[d][1 + d] for d in range(dim))
        heat = self.mu * GAMMA / PR
        out = []
        for c in range(dim):
            tau = [self.mu * (2.0 * grads[c][1 + c] - 2.0 / 3.0 * div) if r == c
                   else self.mu * (grads[c][1 + r] + grads[r][1 + c]) for r in range(dim)]
            cv_dT = (grads[c][-1] - p / rho * grads[c][0]) / ((GAMMA - 1.0) * rho)
            out.append(torch.stack([torch.zeros_like(tau[0])] + tau + [sum(x * t for x, t in zip(v, tau)) + heat * cv_dT]))
        return out
