"""Timed cases of the SIMPLE solver, through its public entry points.

A case is one call pattern of a user's program on one mesh:

  run       a number of outer iterations from a given state (set the fields,
            iterate, read u, v, w, p back): the lid-driven cavity (2-D, 3-D,
            distorted, heated and unsteady) and the k-epsilon backward-facing
            step, with the solver forms that bench.py names
  ensemble  a batch of uneven cavities advanced together (Ensemble.run)
  solve     one linear system alone (SolveEquation), for hosts that assemble
            their own matrices
  net       forward and backward pass of the network behind the learned p'
            guess (nn_eval)

The solver handle (mesh, connectivity, hierarchy) is kept between calls, as a
program that runs one mesh many times keeps it; every pass starts from the
state's own inputs, so passes do not depend on one another.
"""
import math

import numpy as np
import torch

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import ensemble as en
from flowsolversourcecode_b200.solver import Solver

# solver forms of bench.py
FORMS = {
    "fp64": dict(solver_mom="sor", solver_cont="amg_bicgs", krylov_tol=1e-8, krylov_maxit=200),
    "fp64_guess": dict(solver_mom="sor", solver_cont="amg_bicgs", krylov_tol=1e-8, krylov_maxit=200, pc_history=4),
    "mixed": dict(solver_mom="sor", solver_cont="amg32_bicgs", krylov_tol=1e-8, krylov_maxit=200,
                  batched_momentum=True),
    "mixed_gs": dict(solver_mom="sor", solver_cont="amg32gs_bicgs", krylov_tol=1e-8, krylov_maxit=200,
                     batched_momentum=True),
}


def listed():
    return [
        # the smallest run: the 64x64 cavity that also runs on the CPU; launches and barriers count
        {"name": "cavity2d_64", "kind": "run", "flow": "cavity", "nx": 64, "nz": 1, "jitter": 0.0, "form": "fp64",
         "iters": 10},
        # an ordinary 3-D run of odd size whose p' solves start from the previous solutions
        {"name": "cavity_55x41_guess", "kind": "run", "flow": "cavity", "nx": 55, "nz": 41, "jitter": 0.0,
         "form": "fp64_guess", "iters": 8},
        # the headline run: 128^3 cavity, every part in FP64 (the largest case)
        {"name": "cavity_128", "kind": "run", "flow": "cavity", "nx": 128, "nz": 128, "jitter": 0.0, "form": "fp64",
         "iters": 5},
        # the same flow with the FP32 preconditioner and the momentum components solved together, odd size
        {"name": "cavity_95_mixed", "kind": "run", "flow": "cavity", "nx": 95, "nz": 95, "jitter": 0.0,
         "form": "mixed", "iters": 6},
        # a non-orthogonal mesh with the Gauss-Seidel-smoothed preconditioner
        {"name": "distorted_73_gs", "kind": "run", "flow": "cavity", "nx": 73, "nz": 73, "jitter": 0.2,
         "form": "mixed_gs", "iters": 6},
        # turbulent channel flow over a step: k-epsilon, wall functions, inlet and outlet
        {"name": "step_256x48x24", "kind": "run", "flow": "step", "nx": 256, "nz": 24, "jitter": 0.0, "form": "fp64",
         "iters": 5},
        # an unsteady heated cavity: two time steps of three outer iterations, temperature included
        {"name": "heated_45x37", "kind": "run", "flow": "heated", "nx": 45, "nz": 37, "jitter": 0.0, "form": "fp64",
         "iters": 3},
        # a parameter study: 12 uneven cavities in one batched run
        {"name": "ensemble_12", "kind": "ensemble", "cases": 12, "lo": 32, "hi": 56, "iters": 10, "launches": 2,
         "spec": 0},
        # one pressure system with the reference's unpreconditioned BiCGSTAB
        {"name": "pressure_bicgs", "kind": "solve", "nx": 73, "ny": 59, "nz": 47, "system": "pressure",
         "solver": "bicgs"},
        # one larger pressure system with the multigrid-preconditioned BiCGSTAB
        {"name": "pressure_amg_bicgs", "kind": "solve", "nx": 101, "ny": 83, "nz": 67, "system": "pressure",
         "solver": "amg_bicgs"},
        # one transport system (momentum, k, epsilon, temperature) by Gauss-Seidel sweeps
        {"name": "transport_sor", "kind": "solve", "nx": 81, "ny": 64, "nz": 50, "system": "transport",
         "solver": "sor"},
        # network of the learned p' guess: outputs, loss and gradient
        {"name": "net_40", "kind": "net", "nx": 40, "ny": 40, "nz": 40},
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["cavity2d", "cavity", "cavity", "cavity", "step", "heated", "ensemble", "solve", "solve", "net"])
    if what == "cavity2d":
        return {"kind": "run", "flow": "cavity", "nx": _logu(rng, 24, 160), "nz": 1, "jitter": 0.0,
                "form": rng.choice(["fp64", "fp64_guess"]), "iters": rng.randint(5, 10)}
    if what == "cavity":
        return {"kind": "run", "flow": "cavity", "nx": _logu(rng, 16, 108), "nz": _logu(rng, 16, 108),
                "jitter": rng.choice([0.0, 0.0, 0.2]), "form": rng.choice(sorted(FORMS)), "iters": rng.randint(3, 5)}
    if what == "step":
        return {"kind": "run", "flow": "step", "nx": 4 * _logu(rng, 12, 72), "nz": _logu(rng, 6, 26), "jitter": 0.0,
                "form": rng.choice(["fp64", "fp64_guess"]), "iters": rng.randint(3, 5)}
    if what == "heated":
        return {"kind": "run", "flow": "heated", "nx": _logu(rng, 12, 70), "nz": _logu(rng, 12, 70), "jitter": 0.0,
                "form": rng.choice(["fp64", "fp64_guess"]), "iters": rng.randint(2, 4)}
    if what == "ensemble":
        return {"kind": "ensemble", "cases": rng.randint(3, 12), "lo": rng.randint(16, 28), "hi": rng.randint(30, 48),
                "iters": rng.randint(4, 10), "launches": rng.randint(2, 4), "spec": rng.randint(1, 99)}
    size = {k: _logu(rng, 12, 72) for k in ("nx", "ny", "nz")}
    if what == "solve":
        system = rng.choice(["pressure", "transport"])
        solvers = ["bicgs", "amg_bicgs", "amg32_bicgs", "gmres"] if system == "pressure" else ["sor", "ilu", "bicgs"]
        return dict(size, kind="solve", system=system, solver=rng.choice(solvers))
    return dict({k: min(v, 48) for k, v in size.items()}, kind="net")


# ------------------------------------------------------------------ inputs
def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _axes(nx, ny, nz):
    """Unit-box coordinates of the cells of an nx*ny*nz box, x fastest."""
    f = [(torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n for n in (nx, ny, nz)]
    z, y, x = torch.meshgrid(f[2], f[1], f[0], indexing="ij")
    return x.reshape(-1), y.reshape(-1), z.reshape(-1)


def _smooth(g, xyz, noise):
    """A few long waves and a little noise: the shape of a developing field."""
    a = torch.rand((6, 7), generator=g, dtype=torch.float64, device="cuda").cpu()
    out = noise * (2.0 * torch.rand(xyz[0].shape, generator=g, dtype=torch.float64, device="cuda") - 1.0)
    for r in a.tolist():
        s = r[0] - 0.5
        for q in range(3):
            s = s * torch.cos(math.pi * (1 + int(3 * r[1 + q])) * xyz[q] + 6.283 * r[4 + q])
        out = out + s
    return out


# ------------------------------------------------------------------ handles
_held = {}


def _handle(case, make):
    """The solver of this case, kept until another case is prepared."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _held:
        for old in _held.values():
            old[0].close()
        _held.clear()
        _held[key] = make()
    return _held[key]


def _make_run(case):
    kw = dict(FORMS[case["form"]])
    n, nz = case["nx"], case["nz"]
    if case["flow"] == "step":
        kw.pop("batched_momentum", None)
        mesh, c = cs.bfs(n, max(6, 3 * (n // 16)), nz, **kw)
    elif case["flow"] == "heated":
        mesh, c = cs.cavity(n, nz=nz, re=400.0, energy=True, conductivity=0.01, unsteady=True,
                            transient_scheme="adamsmoulton", dt=0.02,
                            thermal={"xmin": ("dirichlet", 1.0), "xmax": ("dirichlet", 0.0)}, **kw)
    elif nz == 1:
        mesh, c = cs.cavity(n, nz=1, re=100.0, **kw)
    else:
        mesh, c = cs.cavity(n, nz=nz, re=1000.0, jitter=case["jitter"], seed=0, conv_scheme="sou", niter_start_hr=1,
                            **kw)
    s = Solver(mesh, c)
    first = {k: _pinned(torch.from_numpy(s.get(k))) for k in ("bu", "bv", "bw", "bp", "bmdot")}
    return s, mesh, c, first


def _make_ensemble(case):
    specs = en.make_specs(case["cases"], seed=case["spec"], edges=(case["lo"], case["hi"]))
    return en.Ensemble([en.build_case(q) for q in specs]), specs


def _make_box(case):
    _, c = cs.cavity(4, krylov_tol=1e-8, krylov_maxit=600)
    mesh = cs.box_mesh(case["nx"], case["ny"], case["nz"])
    return (Solver(mesh, c),)


def _cavity_fields(g, n, nz):
    x, y, z = _axes(n, n, nz)
    wall = 16.0 * x * (1.0 - x) * y * (1.0 - y) * (4.0 * z * (1.0 - z) if nz > 1 else 1.0)
    out = {k: 0.3 * wall * _smooth(g, (x, y, z), 1e-3) for k in ("u", "v", "w")}
    if nz == 1:
        out["w"] = torch.zeros_like(x)
    out["p"] = 0.05 * _smooth(g, (x, y, z), 1e-4)
    return out


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "run":
        s, mesh, c, first = _handle(case, lambda: _make_run(case))
        put = dict(first)
        if case["flow"] == "step":
            ini = cs.bfs_initial_state(mesh, c, seed=int(seed))
            put.update({k: _pinned(torch.from_numpy(v)) for k, v in ini.items()})
            noise = 0.02 * (2.0 * torch.rand((4, s.N), generator=g, dtype=torch.float64, device="cuda") - 1.0)
            put.update({"u": _pinned(1.0 + noise[0]), "v": _pinned(noise[1]), "w": _pinned(noise[2]),
                        "p": _pinned(noise[3])})
            zero = torch.zeros(s.get("utau").shape[0], dtype=torch.float64)
            put.update({"utau": _pinned(zero), "yplus": _pinned(zero)})
        else:
            put.update({k: _pinned(v) for k, v in _cavity_fields(g, case["nx"], case["nz"]).items()})
        if case["flow"] == "heated":
            xyz = _axes(case["nx"], case["nx"], case["nz"])
            put["temp"] = _pinned(1.0 - xyz[0] + 0.1 * _smooth(g, xyz, 1e-3))
            put["btemp"] = _pinned(torch.from_numpy(first["bu"] * 0.0))
            old = torch.zeros((7, s.N), dtype=torch.float64, device="cuda")
            for q, k in ((0, "u"), (1, "v"), (2, "w"), (3, "p"), (6, "temp")):
                old[q] = torch.from_numpy(put[k]).cuda()
            put["old"] = put["oldold"] = _pinned(old.reshape(-1))
            put["bold"] = _pinned(torch.zeros(7 * s.B, dtype=torch.float64))
        return {"case": case, "solver": s, "put": put, "guess": c.pc_history}
    if case["kind"] == "ensemble":
        e, specs = _handle(case, lambda: _make_ensemble(case))
        puts = []
        for q, s in zip(specs, e.solvers):
            f = {k: _pinned(q.lid * v) for k, v in _cavity_fields(g, q.edge, q.edge).items()}
            f["bp"] = _pinned(torch.zeros(s.B, dtype=torch.float64))
            puts.append(f)
        return {"case": case, "ensemble": e, "puts": puts}
    (s,) = _handle(case, lambda: _make_box(case))
    con = s.connectivity()
    cn = torch.from_numpy(con["cn"].reshape(s.W, s.N)).cuda().long()
    if case["kind"] == "solve":
        ac, anb, x = _system(case, cn, g)
        b = ac * x
        for j in range(s.W):
            b = b + torch.where(cn[j] >= 0, anb[j] * x[cn[j].clamp(min=0)], 0.0)
        return {"case": case, "solver": s, "ac": _pinned(ac), "anb": _pinned(anb.reshape(-1)), "bc": _pinned(b),
                "zero": _pinned(torch.zeros(s.N, dtype=torch.float64))}
    theta, feat, face, target = _net_inputs(case, g)
    wgt = torch.zeros((s.W, s.N), dtype=torch.float32, device="cuda")
    i = torch.arange(s.N, device="cuda")
    step = (1, case["nx"], case["nx"] * case["ny"])
    for j in range(s.W):
        d = (cn[j] - i).abs()
        for q in range(3):
            on = (cn[j] >= 0) & (d == step[q])
            wgt[j] = torch.where(on, face[q][torch.minimum(cn[j].clamp(min=0), i)], wgt[j])
    s.nn_create(0, seed=1)
    s.nn_params(set=theta.cpu().numpy())
    return {"case": case, "solver": s, "theta": theta.cpu().numpy(), "x": _pinned(feat), "wgt": _pinned(wgt.reshape(-1)),
            "target": _pinned(target)}


def _solution(case, g):
    return _smooth(g, _axes(case["nx"], case["ny"], case["nz"]), 1e-3)


def _system(case, cn, g):
    """Matrix of a pressure-correction (symmetric, fixed at x = 1) or a
    transport equation (upwind, under-relaxed) on the box, and its solution."""
    x = _solution(case, g)
    n = x.shape[0]
    dims = (case["nx"], case["ny"], case["nz"])
    step = (1, dims[0], dims[0] * dims[1])
    area = (dims[0] ** 2, dims[1] ** 2, dims[2] ** 2)
    i = torch.arange(n, device="cuda")
    rnd = torch.rand((2, 3, n), generator=g, dtype=torch.float64, device="cuda")
    anb = torch.zeros(cn.shape, dtype=torch.float64, device="cuda")
    top = max(area)
    for j in range(cn.shape[0]):
        d = cn[j] - i
        for q in range(3):
            on = (cn[j] >= 0) & (d.abs() == step[q])
            f = torch.minimum(cn[j].clamp(min=0), i)
            coef = (area[q] / top) * (0.6 + 0.8 * rnd[0, q][f])
            if case["system"] == "transport":
                flow = 2.0 * (rnd[1, q][f] - 0.4) * torch.sign(d).double()
                coef = 0.5 * coef + (-flow).clamp(min=0.0)
            anb[j] = torch.where(on, -coef, anb[j])
    ac = -anb.sum(dim=0)
    if case["system"] == "pressure":
        ac = ac + torch.where(i % dims[0] == dims[0] - 1, 2.0 * area[0] / top, 0.0)
    else:
        ac = (ac + 0.02) / 0.7
    return ac, anb, x


def _net_inputs(case, g):
    n = case["nx"] * case["ny"] * case["nz"]
    theta = 0.12 * torch.randn(33665, generator=g, dtype=torch.float32, device="cuda")
    feat = torch.randn((n, 8), generator=g, dtype=torch.float32, device="cuda")
    feat[:, 7] = 1.0
    face = 0.05 + 0.2 * torch.rand((3, n), generator=g, dtype=torch.float32, device="cuda")
    t = _smooth(g, _axes(case["nx"], case["ny"], case["nz"]), 1e-3)
    return theta, feat, face, ((t - t.mean()) / t.std()).float()


# ------------------------------------------------------------------ one pass
def _load(s, put, guess):
    s.set_iteration(0)
    if guess:
        s.set_pc_history(guess)
    for k, v in put.items():
        s.set(k, v)
    s.initialize_mdot()


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        s = state["solver"]
        _load(s, state["put"], state["guess"])
        if case["flow"] == "heated":
            s.set_time_state(0.0, 0.02, 0.02, 0.02, 0)
            for _ in range(2):
                s.run_time_step(case["iters"], tol=0.0)
        else:
            s.run(case["iters"], tol=0.0)
        names = ["u", "v", "w", "p"] + (["tke", "ted"] if case["flow"] == "step" else [])
        names += ["temp"] if case["flow"] == "heated" else []
        return {k: s.get(k) for k in names}
    if case["kind"] == "ensemble":
        e = state["ensemble"]
        for s, f in zip(e.solvers, state["puts"]):
            _load(s, f, 4)
        e.run(case["iters"], case["launches"], batched=True)
        return [{k: s.get(k) for k in ("u", "v", "w", "p")} for s in e.solvers]
    s = state["solver"]
    if case["kind"] == "solve":
        s.set("ac", state["ac"])
        s.set("anb", state["anb"])
        s.set("bc", state["bc"])
        s.set("kx", state["zero"])
        s.set("pc", state["zero"])
        s.SolveEquation("pressc", *_target(case), case["solver"])
        return {"x": s.get("pc")}
    s.nn_params(set=state["theta"])
    return s.nn_eval(state["x"], state["wgt"], state["target"])


def _target(case):
    """(residual reduction, most iterations) of the solver; the Krylov solvers
    take theirs from the case (1e-8 within 600)."""
    return (0.001, 100) if case["system"] == "pressure" else (0.01, 30)


# ------------------------------------------------------------------ bounds and 64-bit values
def _cells(case):
    if case["kind"] == "run":
        n = case["nx"]
        if case["flow"] == "step":
            return n * max(6, 3 * (n // 16)) * case["nz"]
        return n * n * case["nz"]
    if case["kind"] == "ensemble":
        return sum(q.cells for q in en.make_specs(case["cases"], seed=case["spec"], edges=(case["lo"], case["hi"])))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Each outer iteration reads the mesh (connectivity and geometry: 150
    bytes a face of three a cell, 100 a cell), the state and each of its
    systems (80 bytes a row) and writes the state once; the passes of the
    linear solvers beyond the first are not counted."""
    n = _cells(case)
    if case["kind"] == "run":
        eqs = {"cavity": 4, "heated": 5, "step": 6}[case["flow"]]
        its = case["iters"] * (2 if case["flow"] == "heated" else 1)
        return {"bytes": its * n * (3 * 150 + 100 + eqs * (80 + 40)), "flops": its * n * eqs * 150}
    if case["kind"] == "ensemble":
        its = case["iters"] * case["launches"]
        return {"bytes": its * n * (3 * 150 + 100 + 4 * 120), "flops": its * n * 600}
    if case["kind"] == "solve":
        return {"bytes": n * (80 + 8 + 8), "flops": n * 13}
    return {"bytes": n * (8 * 4 + 6 * 8 + 4 + 4) + 2 * 33665 * 4, "flops": 6 * n * (8 * 64 + 4 * 128 * 64 + 64)}


def exact(case, seed):
    g = _gen(seed)
    if case["kind"] == "solve":
        return {"x": _solution(case, g).cpu()}
    if case["kind"] != "net":
        return None
    theta, feat, face, target = _net_inputs(case, g)
    th = theta.double().requires_grad_(True)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz

    def neighbours(h):
        v = h.reshape(nz, ny, nx, 64)
        out = torch.zeros_like(v)
        for q, dim in ((0, 2), (1, 1), (2, 0)):
            m = v.shape[dim]
            w = face[q].double().reshape(nz, ny, nx, 1).narrow(dim, 0, m - 1)
            lo = torch.nn.functional.pad(w * v.narrow(dim, 1, m - 1), [0, 0] * (3 - dim) + [0, 1])
            hi = torch.nn.functional.pad(w * v.narrow(dim, 0, m - 1), [0, 0] * (3 - dim) + [1, 0])
            out = out + lo + hi
        return out.reshape(n, 64)

    at = 0

    def take(*shape):
        nonlocal at
        k = math.prod(shape)
        at += k
        return th[at - k:at].reshape(shape)

    w, b = take(8, 64), take(64)
    h = torch.relu(feat.double() @ w + b)
    for _ in range(4):
        w, b = take(128, 64), take(64)
        h = h + torch.relu(torch.cat([h, neighbours(h)], dim=1) @ w + b)
    w, b = take(64), take(1)
    y = h @ w + b
    t = target.double()
    loss = ((y - y.mean() - t) ** 2).sum() / (t * t).sum()
    loss.backward()
    return {"y": y.detach().cpu(), "loss": float(loss), "grad": th.grad.cpu()}
