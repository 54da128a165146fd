"""The work that a user of this framework has it do, as cases that can be timed.

A flow case is a run from a stored state: the user's arrays go to the device, the solver takes a number of
physical steps there and the conserved variables come back (scfd_upload / scfd_prepare / scfd_run /
scfd_download through shared_cfd_b200.solver.Solver). The other cases are the chemical equilibrium of a batch
of cells, a batch of 0-D reactors, and the gradient of a boundary force by the discrete adjoint.
"""
import collections
import copy
import ctypes
import functools
import math

import numpy as np
import torch

from shared_cfd_b200 import abi, cases, cea
from shared_cfd_b200.adjoint import adjoint_run
from shared_cfd_b200.reactors import Reactors
from shared_cfd_b200.solver import Solver

RU = 8.3144621  # J/(mol K), as the CEA tables are used with


def listed():
    return [
        # the shock tube that every new user runs first: small kernels, hundreds of explicit steps
        dict(name="sod_400x4", kind="sod", ni=400, nj=4, steps=200, mixed=False),
        # a laminar flat plate on its way to the steady state: LU-SGS with a local time step
        dict(name="plate_256x128", kind="plate", ni=256, nj=128, steps=100, mixed=False),
        # the same on a grid of odd sizes, FP32 fluxes and sweeps
        dict(name="plate_301x173_mixed", kind="plate", ni=301, nj=173, steps=60, mixed=True),
        # a low-Mach unsteady flow with the preconditioned dual time
        dict(name="dual_64", kind="dual", n=64, inner=20, steps=3, mixed=False),
        # a coarse reacting step, as in a check of a new set-up
        dict(name="reacting_1/32", kind="reacting", scale=1.0 / 32.0, inner=20, steps=4, mixed=False),
        # the reacting step on a middling grid with ragged rows (148 x 148 and 148 x 74)
        dict(name="reacting_0.29", kind="reacting", scale=0.29, inner=20, steps=3, mixed=False),
        # production: the full reacting step, 786 432 cells, in FP64 and in mixed precision
        dict(name="reacting_full", kind="reacting", scale=1.0, inner=20, steps=4, mixed=False),
        dict(name="reacting_full_mixed", kind="reacting", scale=1.0, inner=20, steps=4, mixed=True),
        # chemical equilibrium of a small odd batch and of a large grid, warm-started as a flow solver does
        dict(name="cea_4099", kind="cea", n=4099),
        dict(name="cea_1m", kind="cea", n=1 << 20),
        # ignition delays of a batch of constant-volume reactors
        dict(name="reactors_8192", kind="reactors", n=8192, t_end=5e-4),
        # the gradient of a wall force with respect to the inflow, 196 608 cells and 300 steps
        dict(name="adjoint_256", kind="adjoint", n=256, steps=300, snapshots=16),
    ]


def _spread(rng, lo, hi):
    """An integer, uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sod", "plate", "dual", "reacting", "reacting", "cea", "reactors", "adjoint"])
    mixed = rng.random() < 0.4
    if kind == "sod":
        return dict(kind=kind, ni=_spread(rng, 100, 4000), nj=_spread(rng, 4, 64), steps=rng.randint(20, 200),
                    mixed=mixed)
    if kind == "plate":
        return dict(kind=kind, ni=_spread(rng, 40, 512), nj=_spread(rng, 40, 300), steps=rng.randint(20, 100),
                    mixed=mixed)
    if kind == "dual":
        return dict(kind=kind, n=_spread(rng, 10, 100), inner=rng.randint(6, 30), steps=rng.randint(2, 4),
                    mixed=mixed)
    if kind == "reacting":
        return dict(kind=kind, scale=round(math.exp(rng.uniform(math.log(1.0 / 32.0), 0.0)), 4),
                    inner=rng.randint(4, 20), steps=rng.randint(2, 4), mixed=mixed)
    if kind == "cea":
        return dict(kind=kind, n=_spread(rng, 256, 1 << 20))
    if kind == "reactors":
        return dict(kind=kind, n=_spread(rng, 64, 8192), t_end=rng.uniform(2e-5, 5e-4))
    return dict(kind=kind, n=_spread(rng, 24, 256), steps=rng.randint(60, 300), snapshots=rng.choice([4, 8, 16]))


# ---------------------------------------------------------------------------
# flow cases
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _grid(kind, a, b, inner):
    """The case before its initial state is disturbed: grid, connectivity, boundaries and tables, which a user
    has in files."""
    if kind == "sod":
        return cases.sod(a, b)
    if kind == "plate":
        return cases.flat_plate(a, b)
    if kind == "dual":
        case = cases.forward_step(0, n=a, scheme=abi.SCHEME_DUAL, viscous=1)
        case.desc.num_internal_loop = inner + 1
        case.desc.cfl_tau = 5.0
        case.desc.res_rate_err = 1e300
        return case
    return cases.reacting_step(scale=a, inner=inner)


def _flow_case(case, seed):
    kind = case["kind"]
    size = {"sod": ("ni", "nj"), "plate": ("ni", "nj"), "dual": ("n", "n"), "reacting": ("scale", "scale")}[kind]
    base = _grid(kind, case[size[0]], case[size[1]], case.get("inner", 0))
    c = copy.copy(base)
    c.desc = abi.Desc.from_buffer_copy(base.desc)
    c.desc.precision = abi.PREC_MIXED if case["mixed"] else abi.PREC_FP64
    c.q, c.w, c.vhi = base.q.copy(), base.w.copy(), base.vhi.copy()
    return cases.perturb(c, seed=seed, amp={"sod": 0.02, "plate": 0.01, "dual": 0.05, "reacting": 0.005}[kind])


def _pinned(a):
    t = torch.from_numpy(a).pin_memory() if torch.cuda.is_available() else torch.from_numpy(a)
    return t.numpy()


def _prepare_flow(case, seed):
    c = _flow_case(case, seed)
    s = {"solver": Solver(c), "steps": case["steps"], "q": _pinned(c.q), "w": _pinned(c.w), "vhi": _pinned(c.vhi),
         "out": _pinned(np.zeros_like(c.q)), "tt": ctypes.c_double(), "mixed": case["mixed"]}
    return s


def _run_flow(s):
    sol = s["solver"]
    sol.upload(s["q"], s["w"], s["vhi"])
    sol.prepare(1)
    sol.run(1, s["steps"])
    sol._check(sol.lib.download(sol.ctx, abi.dptr(s["out"]), None, None, ctypes.byref(s["tt"])), "download")
    q = torch.from_numpy(s["out"])
    # the mixed path's state is good to single precision, and is kept as that
    return {"q": q.float() if s["mixed"] else q, "tt": s["tt"].value}


# ---------------------------------------------------------------------------
# chemical equilibrium, reactors, adjoint
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _cea_data():
    return cea.h2_air_data()


def _cea_states(info, n, seed):
    rho, Y, e, T = cea.random_states(info, n, seed=seed)
    return rho, Y, e, e + 0.01 * np.abs(e), T


def _prepare_cea(case, seed):
    """Cells solved once; each pass then moves every cell's energy by 1 % and solves from the last T and n, as the
    flow model does from step to step."""
    g = cea.Cea(_cea_data())
    rho, Y, e0, e1, T = _cea_states(g.info(), case["n"], seed)
    n, dev = case["n"], torch.device("cuda", torch.cuda.current_device())

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    def new(*shape):
        return torch.empty(shape, dtype=torch.float64, device=dev)
    s = {"cea": g, "rho": t(rho), "Y": t(Y), "e": collections.deque([t(e1), t(e0)]), "T": t(T),
         "n": t(g.initial_n(n)), "mwave": new(n), "kappa": new(n), "mu": new(n), "Yv": new(g.ns, n),
         "vhi": new(g.ns, n), "DHi": new(2, n), "iters": torch.empty(n, dtype=torch.int32, device=dev)}
    g.solve_device(s["rho"], s["Y"], s["e"][1], s["T"], s["n"])
    return s


CEA_OUT = ("T", "n", "mwave", "kappa", "mu", "Yv", "vhi", "DHi", "iters")


def _run_cea(s):
    e = s["e"][0]
    s["e"].rotate(-1)
    s["cea"].solve_device(s["rho"], s["Y"], e, *[s[k] for k in CEA_OUT])
    return {k: s[k] for k in CEA_OUT}


def _prepare_reactors(case, seed):
    m, chem, T0, vrho0, _ = cases.reactor_batch(case["n"], seed=seed)
    return {"reactors": Reactors(chem, case["n"]), "T0": T0, "vrho0": vrho0, "t_end": case["t_end"]}


def _run_reactors(s):
    out = s["reactors"].run(s["T0"], s["vrho0"], s["t_end"])
    if out.pop("status"):
        raise RuntimeError("reactors failed")
    return out


@functools.lru_cache(maxsize=4)
def _channel(n):
    return cases.adjoint_channel(n=n, seed=0)


def _adjoint_case(case, seed):
    base = _channel(case["n"])
    c = copy.copy(base)
    for p in range(2):
        c.q, c.w, c.vhi = c.q.copy(), c.w.copy(), c.vhi.copy()
        snd = math.sqrt(1.4 * 1e5 / 1.2)
        cases.fill_all(c, p, *cases.ideal_state(c, 1.2, 0.5 * snd, 0.0, 1e5))
    return cases.perturb(c, seed=seed, amp=0.02)


def _window(steps):
    return 2 * steps // 3, steps - 1


def _prepare_adjoint(case, seed):
    c = _adjoint_case(case, seed)
    return {"solver": Solver(c), "q": _pinned(c.q), "w": _pinned(c.w), "vhi": _pinned(c.vhi), "steps": case["steps"],
            "snapshots": case["snapshots"], "window": _window(case["steps"])}


def _run_adjoint(s):
    s["solver"].upload(s["q"], s["w"], s["vhi"])
    J, grad, _ = adjoint_run(s["solver"], s["steps"], 2, s["window"], 0, snapshots=s["snapshots"])
    return {"J": J, "grad": grad}


def prepare(case, seed):
    kind = case["kind"]
    f = {"cea": _prepare_cea, "reactors": _prepare_reactors, "adjoint": _prepare_adjoint}.get(kind, _prepare_flow)
    s = f(case, seed)
    s["run"] = {"cea": _run_cea, "reactors": _run_reactors, "adjoint": _run_adjoint}.get(kind, _run_flow)
    return s


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the caller's arrays read once and the results written once. Flops: estimates per cell of the
    arithmetic itself (a quotient or root counted once, exp and log as 20)."""
    kind = case["kind"]
    if kind == "cea":
        # 112 B in, 268 B out; about 2.6 Newton iterations of 9 species (exp, log, two 9-term dots) and a 4 x 4 LU
        return {"bytes": 380.0 * case["n"], "flops": 2.6 * (9 * 110 + 200) * case["n"] + 9 * 9 * 8 * case["n"]}
    if kind == "reactors":
        # about 4 evaluations of 19 reactions and 9 species per call of 1 microsecond
        return {"bytes": 8.0 * case["n"] * 25, "flops": 4 * (45 * 9 + 60 * 19) * case["n"] * case["t_end"] / 1e-6}
    if kind == "adjoint":
        cells = 3 * case["n"] ** 2
        return {"bytes": 8.0 * 14 * cells, "flops": cells * case["steps"] * (550.0 + 1650.0)}
    D = 12 if kind == "reacting" else 4
    if kind in ("sod", "plate"):
        cells, its = case["ni"] * case["nj"], case["steps"]
        flops = cells * its * (600.0 if kind == "sod" else 1200.0)
    elif kind == "dual":
        cells, its = 3 * case["n"] ** 2, case["steps"] * case["inner"]
        flops = cells * its * 1400.0
    else:
        n5, n2 = (max(4, int(round(k * case["scale"]))) for k in (512, 256))
        cells = 2 * n5 * (n5 + n2)
        # per inner iteration: two faces, thermodynamics and transport, two sweeps; once per step the chemistry
        flops = cells * case["steps"] * (case["inner"] * 3500.0 + 6000.0)
    return {"bytes": 8.0 * cells * (D + (D + 5) + (D - 3) + D), "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, without the framework's code
# ---------------------------------------------------------------------------
def _faces(w, phi, km):
    """Left and right states at the faces between the inner cells of w[..., 2 ghosts + cells + 2 ghosts]."""
    d = w[..., 1:] - w[..., :-1]
    lo, up = d[..., :-1], d[..., 1:]
    s = 2.0 * up * lo / (up * up + lo * lo + 1e-300)
    du = 0.5 * s * ((1.0 + km * s) * up + (1.0 - km * s) * lo)
    dl = 0.5 * s * ((1.0 + km * s) * lo + (1.0 - km * s) * up)
    c = w[..., 1:-1]
    return (c + 0.5 * phi * du)[..., :-1], (c - 0.5 * phi * dl)[..., 1:]


def _abs(x):
    """|x| with the slope 1 at 0, as the framework's reverse takes it (wall faces have no mass flux at all)."""
    return torch.where(x >= 0.0, x, -x)


def _slau(l, r, normal):
    """SLAU flux of (rho, rho u, rho v, E) through faces with the unit normal along x (0) or y (1); l, r hold
    rho, u, v, p, Y, gamma, h_t."""
    rl, ul, vl, pl, yl, gl, hl = l
    rr, ur, vr, pr, yr, gr, hr = r
    a = 0.5 * (torch.sqrt(gr * pr / rr) + torch.sqrt(gl * pl / rl))
    unl, unr = (ul, ur) if normal == 0 else (vl, vr)
    ml, mr = unl / a, unr / a
    mt = torch.clamp(torch.sqrt(0.5 * (ul * ul + vl * vl + ur * ur + vr * vr)) / a, max=1.0)
    chi = (1.0 - mt) ** 2
    g = -torch.clamp(ml, -1.0, 0.0) * torch.clamp(mr, 0.0, 1.0)
    ub = (_abs(unr) * rr + _abs(unl) * rl) / (rr + rl)
    m = 0.5 * (rl * (unl + (1.0 - g) * ub + g * _abs(unl)) + rr * (unr - (1.0 - g) * ub - g * _abs(unr)) -
               chi / a * (pr - pl))
    br = torch.where(mr.abs() < 1.0, 0.25 * (2.0 + mr) * (mr - 1.0) ** 2, 0.5 * (1.0 - torch.sign(mr)))
    bl = torch.where(ml.abs() < 1.0, 0.25 * (2.0 - ml) * (ml + 1.0) ** 2, 0.5 * (1.0 + torch.sign(ml)))
    pb = 0.5 * (pr + pl)
    p = pb + 0.5 * (bl - br) * (pl - pr) + (1.0 - chi) * (br + bl - 1.0) * pb
    up, dn = 0.5 * (m + _abs(m)), 0.5 * (m - _abs(m))
    f = [up * yl + dn * yr, up * ul + dn * ur, up * vl + dn * vr, up * hl + dn * hr]
    f[1 + normal] = f[1 + normal] + p
    return torch.stack(f)


def _primitive(q, kg, rgas):
    rho, u, v = q[0], q[1] / q[0], q[2] / q[0]
    p = (kg - 1.0) * (q[3] - 0.5 * rho * (u * u + v * v))
    one = torch.ones_like(rho)
    return torch.stack([rho, u, v, p, one, kg * one, (q[3] + p) / rho])


def _residual(w, lo, hi, wall, dx, dy, d):
    """Sum of the fluxes into the cells of w[k, j, i]; lo, hi: the ghost states beyond the first and last column;
    wall: slip walls below and above, else zero gradient."""
    def ghost(g):
        return g[:, :, None].expand(-1, -1, 2)
    wi = torch.cat([ghost(lo), w, ghost(hi)], dim=2)
    flip = torch.tensor([1.0, 1.0, -1.0 if wall else 1.0, 1.0, 1.0, 1.0, 1.0], dtype=w.dtype, device=w.device)
    b, t = w[:, 0] * flip[:, None], w[:, -1] * flip[:, None]
    wj = torch.cat([b[:, None], b[:, None], w, t[:, None], t[:, None]], dim=1).transpose(1, 2)
    fi = _slau(*_faces(wi, d.phi_mus, d.k_mus), 0) * dy[None, :, None]
    fj = (_slau(*_faces(wj, d.phi_mus, d.k_mus), 1) * dx[None, :, None]).transpose(1, 2)
    return fi[..., :-1] - fi[..., 1:] + fj[:, :-1] - fj[:, 1:]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _widths(c):
    """Cell widths of the row of blocks c, joined along i."""
    f = functools.partial(torch.tensor, dtype=torch.float64, device=_device())
    return (f(np.concatenate([np.diff(xh[:, 0]) for xh, _ in c.planes])), f(np.diff(c.planes[0][1][0])))


def _exact_sod(case, seed):
    c = _flow_case(case, seed)
    d, (dx, dy) = c.desc, _widths(c)
    vol = dy[:, None] * dx[None, :]
    q = torch.tensor(np.moveaxis(c.interior(c.q, 0), 2, 0).copy(), device=_device())
    tt = torch.zeros((), dtype=torch.float64, device=_device())
    for _ in range(case["steps"]):
        w = _primitive(q, d.kappa, d.rgas)
        a = torch.sqrt(d.kappa * w[3] / w[0])
        dt = (d.cfl * vol / (2.0 * ((w[1].abs() + a) * dy[:, None] + (w[2].abs() + a) * dx[None, :]))).min()
        q = q + dt / vol * _residual(w, w[:, :, 0], w[:, :, -1], False, dx, dy, d)
        tt = tt + dt
    out = c.q.copy()
    c.interior(out, 0)[...] = np.moveaxis(q.cpu().numpy(), 0, 2)
    return {"q": torch.from_numpy(out), "tt": float(tt)}


def _exact_adjoint(case, seed):
    """Backpropagation through the plain steps, recomputing each; the two blocks joined to one row."""
    from torch.utils.checkpoint import checkpoint
    c = _adjoint_case(case, seed)
    d, (dx, dy) = c.desc, _widths(c)
    vol, (first, last) = dy[:, None] * dx[None, :], _window(case["steps"])
    q = torch.tensor(np.concatenate([np.moveaxis(c.interior(c.q, p), 2, 0) for p in range(2)], axis=2).copy(),
                     device=_device())
    values = torch.tensor(c.bcs[0].value[:], dtype=torch.float64, device=_device(), requires_grad=True)
    wall = slice(0, case["n"])  # the lower wall of the first block

    def step(q, values):
        w = _primitive(q, d.kappa, d.rgas)
        lo = torch.stack([values[k] for k in (0, 1, 2, 3, 4, 5, 6)])[:, None].expand(-1, w.shape[1])
        return q + d.dt_fixed / vol * _residual(w, lo, w[:, :, -1], True, dx, dy, d)
    J = torch.zeros((), dtype=torch.float64, device=_device())
    for n in range(last + 1):
        if n >= first:
            J = J + (dx[wall] * _primitive(q, d.kappa, d.rgas)[3, 0, wall]).sum()
        if n < last:
            q = checkpoint(step, q, values, use_reentrant=False)
    (g,) = torch.autograd.grad(J, values)
    return {"J": J.item(), "grad": g.cpu().numpy()}


def _exact_cea(case, seed):
    """Newton's method on the element potentials and ln T from the moles' logarithms, to rounding."""
    data, dev = _cea_data(), _device()
    with cea.Cea(data) as g:
        info = g.info()
    rho, Y, _, e, _ = _cea_states(info, case["n"], seed)
    ne, ns = data.ne, data.ns
    f = functools.partial(torch.tensor, dtype=torch.float64, device=dev)
    rho, Y, e = f(rho), f(Y), f(e)
    b = f(info.fuel.b0[:ne])[:, None] * Y[0] + f(info.oxidizer.b0[:ne])[:, None] * Y[1]
    A = f(np.frombuffer(data.ac).reshape(abi.CEA_MAX_SPECIES, -1)[:ns, :ne].T.copy())
    co = f(np.frombuffer(data.co).reshape(abi.CEA_MAX_SPECIES, abi.CEA_MAX_SECTIONS, 9)[:ns].copy())
    tr = f(np.frombuffer(data.trange).reshape(abi.CEA_MAX_SPECIES, abi.CEA_MAX_SECTIONS, 2)[:ns].copy())
    nsec = list(data.nsec)[:ns]

    def thermo(T):
        """cp/R, h/RT and s/R of every species."""
        lt, one, z = torch.log(T), torch.ones_like(T), torch.zeros_like(T)
        pc = torch.stack([T ** -2, 1 / T, one, T, T ** 2, T ** 3, T ** 4, z, z])
        ph = torch.stack([-T ** -2, lt / T, one, T / 2, T ** 2 / 3, T ** 3 / 4, T ** 4 / 5, 1 / T, z])
        ps = torch.stack([-0.5 * T ** -2, -1 / T, lt, T, T ** 2 / 2, T ** 3 / 3, T ** 4 / 4, z, one])
        out = []
        for j in range(ns):
            sec = torch.zeros_like(T, dtype=torch.long)
            for k in range(1, nsec[j]):
                sec = torch.where(T >= tr[j, k, 0], k, sec)
            cj = co[j][sec].T
            out.append(torch.stack([(cj * x).sum(0) for x in (pc, ph, ps)]))
        return torch.stack(out).unbind(1)

    T = torch.full_like(e, 2000.0)
    ln = torch.log((b.sum(0) / ns)[None, :]).expand(ns, -1).clone()
    for it in range(150):
        n = torch.exp(ln)
        cp, h, s = thermo(T)
        u, mu = h - 1.0, h - s + ln + torch.log(rho * RU * T / 1e5)
        # dln n_j = sum_i a_ij pi_i + u_j dln T - mu_j; element and energy balances close the system
        M = torch.zeros(case["n"], ne + 1, ne + 1, dtype=torch.float64, device=dev)
        r = torch.zeros(case["n"], ne + 1, dtype=torch.float64, device=dev)
        for i in range(ne):
            for k in range(ne):
                M[:, i, k] = (A[i][:, None] * A[k][:, None] * n).sum(0)
            M[:, i, ne] = M[:, ne, i] = (A[i][:, None] * n * u).sum(0)
            r[:, i] = b[i] - (A[i][:, None] * n * (1.0 - mu)).sum(0)
        M[:, ne, ne] = (n * (u * u + cp - 1.0)).sum(0)
        r[:, ne] = e / (RU * T) - (n * u * (1.0 - mu)).sum(0)
        scale = 1.0 / torch.sqrt(torch.diagonal(M, dim1=1, dim2=2))
        x = torch.linalg.solve(M * scale[:, :, None] * scale[:, None, :], r * scale) * scale
        dl = A.T @ x[:, :ne].T + u * x[:, ne] - mu
        size = torch.maximum(5.0 * x[:, ne].abs(), torch.where(ln > -18.4, dl.abs(), dl.clamp(min=0.0)).max(0).values)
        lam = torch.clamp(2.0 / size.clamp(min=1e-30), max=1.0)
        ln = (ln + lam * dl).clamp(min=-90.0)
        T = T * torch.exp(lam * x[:, ne])
        if it > 3 and float(size.max()) < 1e-10:
            break
    return {**dict.fromkeys(CEA_OUT), "T": T, "n": torch.exp(ln)}


def exact(case, seed):
    """The flow cases with implicit sweeps or chemistry, and the reactors, have none: plain code for them would be
    the whole solver again, cell by cell."""
    if case["kind"] == "sod" and not case["mixed"]:
        return _exact_sod(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "cea":
        return _exact_cea(case, seed)
    return None
