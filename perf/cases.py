"""Performance cases: the work a program that uses zoomy_b200 has it do.

Each kind of case goes through the public entry points of the host package as
a user's program calls them:

* ``solve``     ``HyperbolicSolver.run_simulation`` to an end time (the host
                polls the control block between batches of steps);
* ``march``     ``HyperbolicSolver.init_march`` + ``launch_steps``: a given
                number of fused steps queued without a host round trip;
* ``step``      the host-driven loop ``compute_timestep`` / ``step`` /
                ``post_step`` (with MOOD: what a coupled or a-posteriori
                limited run does);
* ``ensemble``  ``Ensemble.init`` + ``launch_steps``: batched independent grids;
* ``tri``       the fused steps on an unstructured triangle mesh;
* ``trimesh``   ``DeviceTriangleMesh`` + ``device_arrays`` from host vertices
                and triangles, the preparation of a mesh a program has read;
* ``chorin``    ``ChorinSolver.run_jit_steps``: predictor, pressure solve,
                corrector;
* ``smoother``  ``LearnedSmoother.apply``: inference of the U-Net smoother;
* ``train``     ``SmootherTrainer.step``: forward, backward and Adam.

A pass starts from the case's initial condition (copied into the working
state, as a parameter study does between its runs), so every pass does the
same work.
"""
import math
import pathlib
import sys

import numpy as np
import torch

_PKG = str(pathlib.Path(__file__).resolve().parents[1] / "zoomy-jax_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import zoomy_b200 as zb  # noqa: E402
from zoomy_b200.ensemble import Ensemble  # noqa: E402
from zoomy_b200.fvm.chorin import ChorinSolver  # noqa: E402
from zoomy_b200.fvm.solver import HyperbolicSolver  # noqa: E402
from zoomy_b200.learned import LearnedSmoother, SmootherTrainer  # noqa: E402
from zoomy_b200.trimesh import DeviceTriangleMesh  # noqa: E402

G = 9.81
EPS = 1e-6                       # wet/dry threshold of the benchmark configurations
SIDES = ("left", "right", "bottom", "top")
KINDS = {"extrapolation": 0, "wall": 1, "periodic": 2}


# ── the cases ───────────────────────────────────────────────────────────────
def _flow(kind, nx, ny, dtype, steps, recon="eta", riemann="hll_hr", limiter="minmod", bc="wall",
          manning=0.0, implicit=False, dry=False, mood=False, order=2):
    return {"kind": kind, "nx": nx, "ny": ny, "dtype": dtype, "steps": steps, "order": order,
            "recon": recon, "riemann": riemann, "limiter": limiter, "bc": bc,
            "manning": manning, "implicit": implicit, "dry": dry, "mood": mood}


def listed():
    return [
        # a whole small simulation, the reference's default float64: launches,
        # polls and latency count
        {"name": "solve_64_f64", **_flow("solve", 64, 64, "float64", 24)},
        # a ragged mid-size river reach: friction, open and closed sides
        {"name": "march_517x389_f32", **_flow("march", 517, 389, "float32", 8, bc="open_x",
                                              manning=0.03, implicit=True)},
        # doubly periodic box, conservative reconstruction (wave studies)
        {"name": "march_600x450_f64_periodic",
         **_flow("march", 600, 450, "float64", 6, recon="conservative", riemann="rusanov",
                 limiter="barth_jespersen", bc="periodic")},
        # the benchmark grid in both precisions
        {"name": "march_2048_f32", **_flow("march", 2048, 2048, "float32", 6)},
        {"name": "march_2048_f64", **_flow("march", 2048, 2048, "float64", 3)},
        # the host-driven loop with MOOD over emerging islands
        {"name": "step_320x200_f64_mood",
         **_flow("step", 320, 200, "float64", 3, manning=0.02, dry=True, mood=True)},
        # batched parameter study, uneven instances
        {"name": "ensemble_64_f32", "kind": "ensemble", "count": 64, "lo": 64, "hi": 512,
         "dtype": "float32", "limiter": "minmod", "steps": 6},
        # unstructured lake with friction
        {"name": "tri_980k_f32", "kind": "tri", "side": 701, "dtype": "float32", "steps": 6,
         "manning": 0.03},
        # reading a mesh in
        {"name": "trimesh_320k", "kind": "trimesh", "side": 401, "dtype": "float32"},
        # projection steps at the benchmark's size and tolerance
        {"name": "chorin_1024_f32", "kind": "chorin", "nx": 1024, "ny": 1024,
         "dtype": "float32", "steps": 2, "time_order": 1},
        # learned smoother: one application on the finest level, one Adam step
        # on a batch of patches
        {"name": "smoother_1024_c24", "kind": "smoother", "nx": 1024, "ny": 1024, "c1": 24,
         "c2": 48},
        {"name": "train_b64_c24", "kind": "train", "batch": 64, "n": 32, "c1": 24, "c2": 48,
         "energy": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "march", "march", "march", "march", "step", "ensemble", "tri",
                       "tri", "trimesh", "chorin", "chorin", "smoother", "train"])
    dtype = rng.choice(["float32", "float64"])
    if kind in ("solve", "march", "step"):
        scheme = rng.choice([("eta", "hll_hr"), ("eta", "hll_hr"), ("eta", "rusanov_hr"),
                             ("conservative", "rusanov"), ("constant", "hll_hr")])
        lim = rng.choice(["minmod", "minmod", "barth_jespersen", "venkatakrishnan"])
        hi = {"solve": 256, "march": 2048, "step": 700}[kind]
        nx = _log_int(rng, 32, hi)
        ny = max(16, min(hi, int(nx * rng.uniform(0.6, 1.6))))
        manning = rng.choice([0.0, 0.0, 0.03])
        return _flow(kind, nx, ny, dtype, {"solve": 16, "march": 3, "step": 2}[kind],
                     recon=scheme[0], riemann=scheme[1], limiter=lim,
                     bc=rng.choice(["wall", "wall", "open", "open_x", "periodic"]),
                     manning=manning, implicit=bool(manning) and rng.random() < 0.5,
                     dry=dtype == "float64" and scheme[0] == "eta" and rng.random() < 0.3,
                     mood=kind == "step" and scheme[0] == "eta" and rng.random() < 0.5,
                     order=1 if scheme[0] == "constant" else 2)
    if kind == "ensemble":
        return {"kind": kind, "count": _log_int(rng, 8, 64), "lo": _log_int(rng, 24, 96),
                "hi": _log_int(rng, 128, 512), "dtype": dtype,
                "limiter": rng.choice(["minmod", "venkatakrishnan"]), "steps": 3}
    if kind == "tri":
        return {"kind": kind, "side": _log_int(rng, 30, 701), "dtype": dtype, "steps": 4,
                "manning": rng.choice([0.0, 0.03])}
    if kind == "trimesh":
        return {"kind": kind, "side": _log_int(rng, 40, 401), "dtype": dtype}
    if kind == "chorin":
        m = _log_int(rng, 2, 32)
        return {"kind": kind, "nx": 32 * m, "ny": 32 * max(2, min(32, int(m * rng.uniform(0.6, 1.6)))),
                "dtype": dtype, "steps": 2, "time_order": rng.choice([1, 1, 2])}
    c1, c2 = rng.choice([(8, 16), (16, 16), (16, 32), (24, 48)])
    if kind == "smoother":
        return {"kind": kind, "nx": 2 * _log_int(rng, 32, 512), "ny": 2 * _log_int(rng, 32, 512),
                "c1": c1, "c2": c2}
    return {"kind": kind, "batch": _log_int(rng, 8, 64), "n": rng.choice([16, 24, 32]), "c1": c1,
            "c2": c2, "energy": rng.random() < 0.5}


# ── inputs ──────────────────────────────────────────────────────────────────
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rnd(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _smooth(x, y, g, n, width):
    """Sum of ``n`` Gaussian bumps of random sign-free height, maximum 1."""
    f = torch.zeros_like(x)
    A, cx, cy, w = _rnd(g, 4, n)
    lo, hi = width
    for a, px, py, s in zip(A.tolist(), cx.tolist(), cy.tolist(), w.tolist()):
        s = lo + (hi - lo) * s
        f += (0.2 + a) * torch.exp(-((x - px) ** 2 + (y - py) ** 2) / (2 * s * s))
    return f / f.max()


def _state(x, y, seed, dry=False, flat=False, height=2.0, noise=1e-3):
    """``(4, C)`` float64 state [b, h, qx, qy] at the points ``x, y`` of the
    unit square: a circular dam break over bumps (islands where ``dry``), with
    1e-3 noise on the level and a gentle current."""
    g = _gen(seed)
    b = torch.zeros_like(x) if flat else (1.15 if dry else 0.7) * _smooth(x, y, g, 16, (0.03, 0.1))
    r = torch.sqrt((x - 0.5) ** 2 + (y - 0.5) ** 2)
    level = torch.where(r < 0.2, height, 1.0)
    level = level + noise * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    h = torch.clamp(level - b, min=0.0)
    px, py = _rnd(g, 2).tolist()
    qx = 0.2 * h * torch.sin(2 * math.pi * (y + px))
    qy = 0.2 * h * torch.sin(2 * math.pi * (x + py))
    return torch.stack([b, h, qx, qy])


def _grid_points(nx, ny, lx=1.0, ly=1.0):
    i = torch.arange(nx, device="cuda", dtype=torch.float64)
    j = torch.arange(ny, device="cuda", dtype=torch.float64)
    x = ((i + 0.5) * (lx / nx))[:, None].expand(nx, ny).reshape(-1)
    y = ((j + 0.5) * (ly / ny))[None, :].expand(nx, ny).reshape(-1)
    return x, y


def _dtype(case):
    return torch.float64 if case["dtype"] == "float64" else torch.float32


def _bc(name):
    per = {"wall": "wwww", "open": "eeee", "open_x": "eeww", "periodic": "pppp"}[name]
    full = {"w": "wall", "e": "extrapolation", "p": "periodic"}
    return {s: full[c] for s, c in zip(SIDES, per)}


def _flow_state(case, seed):
    x, y = _grid_points(case["nx"], case["ny"])
    return _state(x, y, seed, dry=case["dry"], flat=case["riemann"] == "rusanov").to(_dtype(case))


# the explicit 2-D CFL law the solver is given
CFL = 0.45


def _dt_scale(case):
    """A bound on the first steps' dt: the end time of a ``solve`` case is a
    multiple of it."""
    dx, dy = 1.0 / case["nx"], 1.0 / case["ny"]
    return CFL * dx * dy / (dx + dy) / 5.5


def _nsm(case, bcs, cells):
    model = zb.ShallowWater2D(g=G, manning_n=case.get("manning", 0.0), wet_dry_eps=EPS,
                              boundary_conditions=bcs, initial_conditions=np.zeros((4, cells)))
    return zb.NumericalSystemModel.from_system_model(
        model, zb.ReconstructionSpec(case.get("order", 2), case.get("limiter", "minmod")),
        case.get("riemann", "hll_hr"))


def _lattice(side, seed):
    """Vertices and triangles (host arrays, as a mesh reader returns them) of
    a jittered lattice with alternating diagonals, cells along a Morton curve."""
    g = _gen(seed)
    n = side
    k = torch.arange(n, device="cuda", dtype=torch.float64) / (n - 1)
    X, Y = torch.meshgrid(k, k, indexing="ij")
    P = torch.stack([X, Y], dim=-1).clone()
    jit = (2 * _rnd(g, n, n, 2) - 1) * (0.25 / (n - 1))
    P[1:-1, 1:-1] += jit[1:-1, 1:-1]
    P = P.reshape(-1, 2)
    i, j = torch.meshgrid(torch.arange(n - 1, device="cuda"), torch.arange(n - 1, device="cuda"),
                          indexing="ij")
    a = (i * n + j).reshape(-1)
    b, c, d = a + n, a + n + 1, a + 1
    odd = ((i + j) % 2 == 1).reshape(-1)
    t1 = torch.where(odd[:, None], torch.stack([a, b, d], 1), torch.stack([a, b, c], 1))
    t2 = torch.where(odd[:, None], torch.stack([b, c, d], 1), torch.stack([a, c, d], 1))
    T = torch.cat([t1, t2])
    q = (P[T].mean(dim=1) * 65535).long()
    key = torch.zeros(len(T), dtype=torch.long, device="cuda")
    for s in range(16):
        key |= ((q[:, 0] >> s) & 1) << (2 * s) | ((q[:, 1] >> s) & 1) << (2 * s + 1)
    T = T[torch.sort(key, stable=True).indices]
    return P.cpu().numpy(), T.to(torch.int32).cpu().numpy()


def _tri_state(P, T, seed):
    c = torch.as_tensor(P, device="cuda")[torch.as_tensor(T, device="cuda").long()].mean(dim=1)
    return _state(c[:, 0].contiguous(), c[:, 1].contiguous(), seed, noise=0.0)


def _ens_sides(case, seed):
    # sides log-uniform over [lo, hi] (an equidistributed sequence: every seed
    # has the same sizes), friction and dam height of each instance random
    g = _gen(seed)
    u = (0.5 + 0.6180339887498949 * np.arange(case["count"])) % 1.0
    sides = np.rint(case["lo"] * (case["hi"] / case["lo"]) ** u).astype(np.int64)
    manning = 0.01 + 0.04 * _rnd(g, case["count"]).cpu().numpy()
    heights = 1.1 + 1.9 * _rnd(g, case["count"]).cpu().numpy()
    return sides, manning, heights


def _ens_state(n, seed, height):
    x, y = _grid_points(n, n)
    return _state(x, y, seed, flat=True, height=float(height))


def _chorin_state(case, seed):
    nx, ny = case["nx"], case["ny"]
    m = max(nx, ny)
    x, y = _grid_points(nx, ny, nx / m, ny / m)
    return _state(x, y, seed).to(_dtype(case)), 1.0 / m


CHORIN_TOL = 1e-8


def _faces(h, lead):
    """Harmonic face means of clip(h, 0.1, 2), the boundary cell's value at
    the sides; ``h (..., nx, ny)``."""
    c = h.clamp(0.1, 2.0)
    fx = 2 * c[..., :-1, :] * c[..., 1:, :] / (c[..., :-1, :] + c[..., 1:, :])
    fy = 2 * c[..., :, :-1] * c[..., :, 1:] / (c[..., :, :-1] + c[..., :, 1:])
    cx = torch.cat([c[..., :1, :], fx, c[..., -1:, :]], dim=-2)
    cy = torch.cat([c[..., :, :1], fy, c[..., :, -1:]], dim=-1)
    return cx.reshape(*lead, *cx.shape[-2:]), cy.reshape(*lead, *cy.shape[-2:])


def _poisson(cx, cy, p, dx):
    """-div(c grad p), p = 0 on the walls; ``p (..., nx, ny)``."""
    px = torch.cat([-p[..., :1, :], p, -p[..., -1:, :]], dim=-2)
    py = torch.cat([-p[..., :, :1], p, -p[..., :, -1:]], dim=-1)
    fx = cx * (px[..., 1:, :] - px[..., :-1, :])
    fy = cy * (py[..., :, 1:] - py[..., :, :-1])
    return -((fx[..., 1:, :] - fx[..., :-1, :]) + (fy[..., :, 1:] - fy[..., :, :-1])) / dx ** 2


def _net_shapes(c1, c2):
    return [(2, c1), (c1, c1), (c1, c2), (c2, c2), (c1 + c2, c1), (c1, 1)]


def _net(case, seed):
    """Network weights as a checkpoint holds them (bf16-representable)."""
    g = torch.Generator().manual_seed(int(seed) + 77)
    ws, bs = [], []
    for ci, co in _net_shapes(case["c1"], case["c2"]):
        ws.append(torch.randn(co * ci * 9, generator=g) * math.sqrt(2.0 / (9 * ci + 9 * co)))
        bs.append(0.05 * torch.randn(co, generator=g))
    return torch.cat(ws).to(torch.bfloat16).float(), torch.cat(bs)


def _smoother(case, seed):
    w, b = _net(case, seed)
    sm = LearnedSmoother(case["c1"], case["c2"], 2.0)
    sm.load_state_dict({"c1": case["c1"], "c2": case["c2"], "cmax": 2.0, "w": w, "b": b})
    return sm


def _patches(case, seed):
    """Residual patches with their coefficients, and the errors behind them."""
    B, n = case["batch"], case["n"]
    g = _gen(seed)
    dx = 1.0 / 256
    k = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    ph = _rnd(g, 4, B, 1, 1)
    fr = 1.0 + 3.0 * _rnd(g, 2, B, 1, 1)
    X, Y = k[None, :, None], k[None, None, :]
    h = 1.0 + 0.8 * torch.sin(6.28 * (fr[0] * X + ph[0])) * torch.cos(6.28 * (Y + ph[1]))
    e = torch.sin(3.14 * X) * torch.sin(3.14 * Y) * torch.cos(6.28 * (fr[1] * X + Y + ph[2]))
    e = (e + 0.05 * torch.randn(B, n, n, generator=g, device="cuda", dtype=torch.float64)) * dx ** 2
    cx, cy = _faces(h, (B,))
    cx, cy, e = cx.float(), cy.float(), e.float()
    r = _poisson(cx.double(), cy.double(), e.double(), dx).float()
    return r.contiguous(), cx.contiguous(), cy.contiguous(), e.contiguous(), dx


def _grid_residual(case, seed):
    nx, ny = case["nx"], case["ny"]
    m = max(nx, ny)
    x, y = _grid_points(nx, ny, nx / m, ny / m)
    S = _state(x, y, seed)
    dx = 1.0 / m
    cx, cy = _faces(S[1].view(nx, ny), ())
    g = _gen(seed + 5)
    noise = torch.randn(2, nx, ny, generator=g, device="cuda", dtype=torch.float64)
    xs = (_smooth(x, y, g, 8, (0.05, 0.2)).view(nx, ny) + 0.1 * noise[0]) * dx ** 2
    f = torch.sin(6.28 * (x + y)).view(nx, ny) + 0.3 * noise[1]
    return (f.float().reshape(-1).contiguous(), xs.float().reshape(-1).contiguous(),
            cx.float().reshape(-1).contiguous(), cy.float().reshape(-1).contiguous(), dx)


# ── prepare / run ───────────────────────────────────────────────────────────
def prepare(case, seed):
    k = case["kind"]
    if k in ("solve", "march", "step"):
        cells = case["nx"] * case["ny"]
        kw = {}
        if case["recon"] == "eta":
            kw = dict(reconstruction_variables="eta", free_surface_h_index=1, eps_wet=EPS)
        end = case["steps"] * _dt_scale(case) if k == "solve" else math.inf
        s = HyperbolicSolver(time_end=end, compute_dt=zb.timestepping.adaptive(CFL, 2),
                             dtype=case["dtype"], mood=case["mood"],
                             implicit_source=case["implicit"], **kw)
        mesh = zb.create_2d((0, 1, 0, 1), case["nx"], case["ny"])
        Q, Qaux = s.setup_simulation(mesh, _nsm(case, _bc(case["bc"]), cells))
        Q0 = _flow_state(case, seed)
        return {"case": case, "solver": s, "Q": Q, "Q0": Q0, "aux0": s.update_qaux(Q0)}
    if k == "ensemble":
        sides, manning, heights = _ens_sides(case, seed)
        E = Ensemble(sides, manning, dtype=case["dtype"], cfl=CFL, wet_dry_eps=EPS, eps_wet=EPS,
                     limiter=case["limiter"])
        E.setup([np.zeros((4, n * n), dtype=np.float32) for n in sides])
        Q0 = torch.cat([_ens_state(int(n), seed + 1 + i, h).reshape(-1).to(_dtype(case))
                        for i, (n, h) in enumerate(zip(sides, heights))])
        return {"case": case, "ens": E, "Q0": Q0}
    if k == "tri":
        P, T = _lattice(case["side"], seed)
        mesh = DeviceTriangleMesh(P, T)
        s = HyperbolicSolver(time_end=math.inf, compute_dt=zb.timestepping.adaptive(CFL, 2),
                             dtype=case["dtype"], reconstruction_variables="eta",
                             free_surface_h_index=1, eps_wet=1e-3, implicit_source=True)
        Q, _ = s.setup_simulation(mesh, _nsm(case, _bc("wall"), mesh.n_cells))
        return {"case": case, "solver": s, "Q": Q, "Q0": _tri_state(P, T, seed).to(_dtype(case))}
    if k == "trimesh":
        P, T = _lattice(case["side"], seed)
        return {"case": case, "P": P, "T": T}
    if k == "chorin":
        Q0, dx = _chorin_state(case, seed)
        nx, ny = case["nx"], case["ny"]
        s = ChorinSolver(pressure_tol=CHORIN_TOL, time_order=case["time_order"],
                         compute_dt=zb.timestepping.adaptive(CFL, 2),
                         reconstruction_variables="eta", free_surface_h_index=1, eps_wet=EPS,
                         dtype=case["dtype"])
        s.setup_simulation(zb.create_2d((0, nx * dx, 0, ny * dx), nx, ny),
                           _nsm(case, _bc("wall"), nx * ny))
        return {"case": case, "solver": s, "Q0": Q0, "dt": 0.2 * dx / 5.0}
    if k == "smoother":
        f, x, cx, cy, dx = _grid_residual(case, seed)
        return {"case": case, "sm": _smoother(case, seed), "f": f, "x": x, "cx": cx, "cy": cy,
                "dx": dx}
    r, cx, cy, e, dx = _patches(case, seed)
    tr = SmootherTrainer(_smoother(case, seed), batch=case["batch"], n=case["n"], lr=1e-4)
    return {"case": case, "tr": tr, "r": r, "cx": cx, "cy": cy, "dx": dx,
            "e": e if case["energy"] else None}


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "solve":
        s, Q = state["solver"], state["Q"]
        Q.copy_(state["Q0"])
        return s.run_simulation(Q, state["aux0"])
    if k in ("march", "tri"):
        s, Q = state["solver"], state["Q"]
        Q.copy_(state["Q0"])
        s.init_march(Q)
        s.launch_steps(Q, case["steps"])
        return Q
    if k == "step":
        s, Q, A = state["solver"], state["Q0"], state["aux0"]
        t = 0.0
        for _ in range(case["steps"]):
            dt = s.compute_timestep(Q, A, time=t)
            Qn = s.step(dt, t, Q, A)
            Q, A = s.post_step(t + dt, dt, Qn, Q, A)
            t += dt
        return Q, A
    if k == "ensemble":
        E = state["ens"]
        E.Q.copy_(state["Q0"])
        E.init()
        E.launch_steps(case["steps"])
        return E.Q
    if k == "trimesh":
        mesh = DeviceTriangleMesh(state["P"], state["T"])
        return mesh.device_arrays(_dtype(case), "cuda", [KINDS["wall"]] * 4)
    if k == "chorin":
        return state["solver"].run_jit_steps(state["dt"], case["steps"], state["Q0"])
    if k == "smoother":
        return state["sm"].apply(case["nx"], case["ny"], state["f"], state["cx"], state["cy"],
                                 state["dx"], x=state["x"])
    tr = state["tr"]
    loss = tr.step(state["r"], state["cx"], state["cy"], state["dx"], target=state["e"])
    return loss, tr.g_w, tr.g_b


# ── the work of a pass ──────────────────────────────────────────────────────
# flops per cell and stage of the finite-volume operator: gradient, bounds and
# limiter of four variables, two faces, the update
_STAGE_FLOPS = {"minmod": 280, "barth_jespersen": 280, "venkatakrishnan": 440}


def work(case):
    k = case["kind"]
    es = 8 if case.get("dtype") == "float64" else 4
    if k in ("solve", "march", "step"):
        cells, steps = case["nx"] * case["ny"], case["steps"]
        # two stages: 4 planes in, 3 out; then 3 + b + 3 in, 3 out
        planes, stages = (17, 2) if case["order"] == 2 else (7, 1)
        if k == "step":
            planes += 3 + 4 + 7          # dt's wave speeds, the aux rows
        return {"bytes": float(cells) * planes * es * steps,
                "flops": float(cells) * _STAGE_FLOPS[case["limiter"]] * stages * steps}
    if k == "ensemble":
        lo, hi = case["lo"], case["hi"]
        mean = (hi * hi - lo * lo) / (2 * math.log(hi / lo))   # of side^2, sides log-uniform
        cells = mean * case["count"]
        return {"bytes": cells * 17 * es * case["steps"],
                "flops": cells * _STAGE_FLOPS[case["limiter"]] * 2 * case["steps"]}
    if k in ("tri", "trimesh"):
        cells = 2.0 * (case["side"] - 1) ** 2
        if k == "tri":
            # state 7 and 10 planes; connectivity and geometry of a cell and of
            # its 1.5 faces once a stage
            per = 17 * es + 2 * (12 + 7 * es + 1.5 * (8 + 4 * es))
            return {"bytes": cells * per * case["steps"],
                    "flops": cells * 500.0 * 2 * case["steps"]}
        return {"bytes": cells * (12 + 8 + 24 + 13 * es + 1.5 * (16 + 7 * es)),
                "flops": cells * 150.0}
    if k == "chorin":
        cells = float(case["nx"]) * case["ny"]
        stages = case["steps"] * case["time_order"]
        # predictor 7 planes; coefficients; right-hand side; a solve that reads
        # its right-hand side and writes the pressure in float64 and, for about
        # eight iterations, passes once over the operator and the residual;
        # corrector
        per = 7 * es + es + 24 + 2 * es + 8 + 16 + 8 * (5 * 8) + 8 + 5 * es
        return {"bytes": cells * per * stages, "flops": cells * stages * (300 + 8 * 150)}
    px = float(case["nx"] * case["ny"]) if k == "smoother" else float(case["batch"] * case["n"] ** 2)
    macs = 0.0
    for (ci, co), s in zip(_net_shapes(case["c1"], case["c2"]), (1, 1, 0.25, 0.25, 1, 1)):
        macs += 9.0 * ci * co * s
    if k == "smoother":
        return {"bytes": px * 20, "flops": 2 * macs * px}
    return {"bytes": px * 16, "flops": 6 * macs * px}


# ── 64-bit values ───────────────────────────────────────────────────────────
def _hinv(h):
    return math.sqrt(2.0) * h / torch.sqrt(h ** 4 + torch.clamp(h, min=EPS) ** 4)


def _clip_min(delta, dpos, dneg):
    one = torch.ones_like(delta)
    p = (dpos / delta.clamp(min=1e-30)).clamp(0, 1)
    n = (dneg / delta.clamp(max=-1e-30)).clamp(0, 1)
    return torch.where(delta > 1e-30, p, torch.where(delta < -1e-30, n, one))


def _venkat(delta, dpos, dneg, e2):
    def side(d, m, sg):
        num = m * m + e2 + 2 * d * m
        den = m * m + 2 * d * d + d * m + e2
        den = den.clamp(min=1e-30) if sg > 0 else den.clamp(max=-1e-30)
        return (sg * num / den).clamp(0, 1)
    one = torch.ones_like(delta)
    return torch.where(delta > 1e-30, side(delta, dpos, 1),
                       torch.where(delta < -1e-30, side(delta, dneg, -1), one))


def _limit(limiter, deltas, dpos, dneg, e2):
    phi = torch.ones_like(dpos)
    for d in deltas:
        c = _venkat(d, dpos, dneg, e2) if limiter == "venkatakrishnan" else _clip_min(d, dpos, dneg)
        phi = torch.minimum(phi, c)
    return phi


def _flux(L, R, n, riemann):
    """Flux through a face with normal ``n = (nx, ny)`` between the traces L
    and R = (b, h, q (2), u (2)): Fh, Fq (2) and the fluctuations of the
    hydrostatic reconstruction."""
    (bL, hL, qL, uL), (bR, hR, qR, uR) = L, R
    nx, ny = n
    unL, unR = uL[0] * nx + uL[1] * ny, uR[0] * nx + uR[1] * ny

    def phys(h, q, un):
        p = 0.5 * G * h * h
        return [q[0] * un + p * nx, q[1] * un + p * ny]
    if riemann == "rusanov":
        s = torch.maximum(unL.abs() + torch.sqrt(G * hL), unR.abs() + torch.sqrt(G * hR))
        fL, fR = phys(hL, qL, unL), phys(hR, qR, unR)
        nL, nR = qL[0] * nx + qL[1] * ny, qR[0] * nx + qR[1] * ny
        Fh = 0.5 * (nL + nR) - 0.5 * s * (hR - hL)
        Fq = [0.5 * (a + b) - 0.5 * s * (y - x) for a, b, x, y in zip(fL, fR, qL, qR)]
        z = torch.zeros_like(Fh)
        return Fh, Fq, z, z
    bs = torch.maximum(bL, bR)
    kL, kR = (hL + bL - bs).clamp(min=0), (hR + bR - bs).clamp(min=0)
    cL, cR = torch.sqrt(G * kL), torch.sqrt(G * kR)
    gL, gR = [kL * u for u in uL], [kR * u for u in uR]
    fL, fR = phys(kL, gL, unL), phys(kR, gR, unR)
    if riemann == "rusanov_hr":
        s = torch.maximum(unL.abs() + cL, unR.abs() + cR)
        Fh = 0.5 * (kL * unL + kR * unR) - 0.5 * s * (kR - kL)
        Fq = [0.5 * (a + b) - 0.5 * s * (y - x) for a, b, x, y in zip(fL, fR, gL, gR)]
    else:
        sl = torch.minimum(unL - cL, unR - cR).clamp(max=0)
        sr = torch.maximum(unL + cL, unR + cR).clamp(min=0)
        den = sr - sl
        inv = torch.where(den > 0, 1.0 / torch.where(den > 0, den, torch.ones_like(den)),
                          torch.zeros_like(den))

        def hll(a, b, x, y):
            return (sr * a - sl * b + sl * sr * (y - x)) * inv
        Fh = hll(kL * unL, kR * unR, kL, kR)
        Fq = [hll(a, b, x, y) for a, b, x, y in zip(fL, fR, gL, gR)]
    return Fh, Fq, 0.5 * G * (hL * hL - kL * kL), -0.5 * G * (hR * hR - kR * kR)


class _Grid:
    """The finite-volume operator on a Cartesian grid, float64 torch."""

    def __init__(self, nx, ny, dx, dy, bc, recon, riemann, limiter, order):
        self.nx, self.ny, self.dx, self.dy, self.bc = nx, ny, dx, dy, bc
        self.recon, self.riemann, self.limiter, self.order = recon, riemann, limiter, order

    def _pad(self, w):
        return torch.nn.functional.pad(w[None], (1, 1, 1, 1))[0]

    def gradient(self, w, ghost):
        """Least-squares gradient over the in-domain 3x3 neighbours; a boundary
        ghost ``ghost[axis][side]`` (value per boundary cell) enters the
        derivative along its axis."""
        nx, ny, dx, dy = self.nx, self.ny, self.dx, self.dy
        m, p = self._pad(torch.ones_like(w)), self._pad(w)
        out = []
        acc = [torch.zeros_like(w) for _ in range(5)]   # sxx sxy syy bx by
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                if a == 0 and b == 0:
                    continue
                ok = m[1 + a:1 + a + nx, 1 + b:1 + b + ny]
                d = (p[1 + a:1 + a + nx, 1 + b:1 + b + ny] - w) * ok
                ox, oy = a * dx, b * dy
                for t, v in zip(acc, (ok * ox * ox, ok * ox * oy, ok * oy * oy, d * ox, d * oy)):
                    t += v
        for axis in (0, 1):
            sxx, sxy, syy, bx, by = (t.clone() for t in acc)
            o = dx if axis == 0 else dy
            for side, sg in ((0, -1.0), (1, 1.0)):
                at = self._edge(axis, side)
                d = ghost[axis][side] - w[at]
                if axis == 0:
                    sxx[at] += o * o
                    bx[at] += d * sg * o
                else:
                    syy[at] += o * o
                    by[at] += d * sg * o
            det = sxx * syy - sxy * sxy
            out.append((syy * bx - sxy * by) / det if axis == 0 else (sxx * by - sxy * bx) / det)
        return out

    def _edge(self, axis, side):
        k = 0 if side == 0 else -1
        return (k, slice(None)) if axis == 0 else (slice(None), k)

    def _kind(self, axis, side):
        return self.bc[SIDES[2 * axis + side]]

    def residual(self, Q, force=None):
        b, h, q = Q[0], Q[1], [Q[2], Q[3]]
        hinv = _hinv(h)
        u = [c * hinv for c in q]
        eta = self.recon == "eta"
        W = [b, b + h, u[0], u[1]] if eta else [b, h, q[0], q[1]]
        if self.order == 2:
            phis, grads = [], []
            e2 = self.dx * self.dy
            for v, w in enumerate(W):
                ghost = []
                for axis in (0, 1):
                    pair = []
                    for side in (0, 1):
                        own = w[self._edge(axis, side)]
                        kind = self._kind(axis, side)
                        if kind == "periodic":
                            own = w[self._edge(axis, 1 - side)]
                        elif kind == "wall" and v == 2 + axis:
                            own = -own
                        pair.append(own)
                    ghost.append(pair)
                gx, gy = self.gradient(w, ghost)
                hi, lo = w.clone(), w.clone()
                for axis in (0, 1):
                    n = w.shape[axis]
                    a, c = w.narrow(axis, 0, n - 1), w.narrow(axis, 1, n - 1)
                    for f, t in ((torch.maximum, hi), (torch.minimum, lo)):
                        t.narrow(axis, 0, n - 1).copy_(f(t.narrow(axis, 0, n - 1), c))
                        t.narrow(axis, 1, n - 1).copy_(f(t.narrow(axis, 1, n - 1), a))
                    for side in (0, 1):
                        at = self._edge(axis, side)
                        gg = 2 * ghost[axis][side] - w[at]
                        hi[at] = torch.maximum(hi[at], gg)
                        lo[at] = torch.minimum(lo[at], gg)
                dX, dY = gx * (0.5 * self.dx), gy * (0.5 * self.dy)
                phis.append(_limit(self.limiter, (dX, -dX, dY, -dY), hi - w, lo - w, e2))
                grads.append((gx, gy))
            if eta:
                wet = (h >= EPS).double()
                phis = [p * wet for p in phis]
                phis = [torch.minimum(p, phis[1]) for p in phis]
            if force is not None:
                phis = [torch.where(force, torch.zeros_like(p), p) for p in phis]
        else:
            z = torch.zeros_like(b)
            phis, grads = [z] * 4, [(z, z)] * 4
        acc = [torch.zeros_like(h) for _ in range(3)]
        for axis in (0, 1):
            o = 0.5 * (self.dx if axis == 0 else self.dy)
            kf = 1.0 / (self.dx if axis == 0 else self.dy)
            traces = []
            for sg in (-1.0, 1.0):      # towards the lower and the upper face
                t = [w + sg * o * p * g[axis] for w, p, g in zip(W, phis, grads)]
                if eta:
                    hf = torch.maximum(t[1], t[0]) - t[0]
                    tr = (t[0], hf, [t[2] * hf, t[3] * hf], [t[2], t[3]])
                else:
                    tr = (t[0], t[1], [t[2], t[3]], [t[2] * hinv, t[3] * hinv])
                traces.append(tr)

            def ghost_of(side):
                at = self._edge(axis, side)
                tr = traces[side]
                pick = (tr[0][at], tr[1][at], [c[at] for c in tr[2]], [c[at] for c in tr[3]])
                kind = self._kind(axis, side)
                if kind == "periodic":
                    far = self._edge(axis, 1 - side)
                    qq = [c[far] for c in q]
                    uu = [c[far] for c in u] if eta else [c * hinv[at] for c in qq]
                    pick = (b[far], h[far], qq, uu)
                elif kind == "wall":
                    qq, uu = list(pick[2]), list(pick[3])
                    qq[axis], uu[axis] = -qq[axis], -uu[axis]
                    pick = (pick[0], pick[1], qq, uu)
                return pick

            def join(tr, gh, side):
                def one(f, g):
                    g = g.unsqueeze(axis)
                    return torch.cat([g, f] if side == 0 else [f, g], dim=axis)
                return (one(tr[0], gh[0]), one(tr[1], gh[1]),
                        [one(a, c) for a, c in zip(tr[2], gh[2])],
                        [one(a, c) for a, c in zip(tr[3], gh[3])])
            # face f lies between cells f - 1 (its upper trace) and f (its lower)
            L, R = join(traces[1], ghost_of(0), 0), join(traces[0], ghost_of(1), 1)
            n = (1.0, 0.0) if axis == 0 else (0.0, 1.0)
            Fh, Fq, Dm, Dp = _flux(L, R, n, self.riemann)
            N = h.shape[axis]
            up, dn = (lambda f: f.narrow(axis, 1, N)), (lambda f: f.narrow(axis, 0, N))
            acc[0] += kf * (up(Fh) - dn(Fh))
            for d in (0, 1):
                acc[1 + d] += kf * (up(Fq[d]) - dn(Fq[d]))
            bed = up(Dm) + dn(Dp)
            if self.order == 2:
                (bl, hl, _, _), (bu, hu, _, _) = traces
                bed = bed + 0.5 * G * (h + hu) * (bu - b) - 0.5 * G * (h + hl) * (bl - b)
            acc[1 + axis] += kf * bed
        return torch.stack([torch.zeros_like(h)] + [-a for a in acc])

    def dt(self, Q):
        hi = _hinv(Q[1])
        c = torch.sqrt(G * Q[1].clamp(min=0))
        lam = torch.maximum((Q[2] * hi).abs() + c, (Q[3] * hi).abs() + c).max()
        return CFL * 2 * self.dx * self.dy / (self.dx + self.dy) / (2 * float(lam))

    def advance(self, Q, dt, force=None):
        Q1 = Q + dt * self.residual(Q, force)
        if self.order == 1:
            return Q1
        return 0.5 * (Q + Q1 + dt * self.residual(Q1, force))

    def step(self, Q, dt, manning=0.0, implicit=False, mood=False):
        Qn = self.advance(Q, dt)
        if mood:
            bad = (Qn[1] < 0) | ~torch.isfinite(Qn).all(dim=0)
            if bool(bad.any()):
                Qn = self.advance(Q, dt, bad)
        return _friction(Qn, Q[1], dt, manning, implicit)

    def aux(self, Q):
        gs = []
        for v in range(4):
            w = Q[v]
            gh = [[w[self._edge(a, s)] for s in (0, 1)] for a in (0, 1)]
            gs.append(self.gradient(w, gh))
        return torch.stack([gs[2][0], gs[1][0], gs[3][1], gs[1][1], gs[0][0], gs[0][1],
                            _hinv(Q[1])])


def _friction(Qn, h0, dt, manning, implicit):
    if manning == 0.0:
        return Qn
    hi = _hinv(h0)
    k = G * manning ** 2 * torch.sqrt(Qn[2] ** 2 + Qn[3] ** 2) * hi ** 2 * hi ** (1.0 / 3.0)
    f = 1.0 / (1.0 + dt * k) if implicit else 1.0 - dt * k
    return torch.stack([Qn[0], Qn[1], Qn[2] * f, Qn[3] * f])


def _exact_flow(case, seed):
    nx, ny = case["nx"], case["ny"]
    g = _Grid(nx, ny, 1.0 / nx, 1.0 / ny, _bc(case["bc"]), case["recon"], case["riemann"],
              case["limiter"], case["order"])
    Q = _flow_state(case, seed).double().view(4, nx, ny)
    t, n = 0.0, 0
    end = case["steps"] * _dt_scale(case) if case["kind"] == "solve" else math.inf
    while (t < end) if case["kind"] == "solve" else (n < case["steps"]):
        dt = min(g.dt(Q), end - t)
        Q = g.step(Q, dt, case["manning"], case["implicit"], case["mood"])
        t, n = t + dt, n + 1
    if case["kind"] == "march":
        return Q.view(4, -1)
    return Q.view(4, -1), g.aux(Q).view(7, -1)


class _Tri:
    """The operator on triangles, cell by cell over their three edges."""

    def __init__(self, P, T):
        P, T = torch.as_tensor(P, device="cuda"), torch.as_tensor(T, device="cuda").long()
        a, b, c = (P[T[:, i]] for i in range(3))
        cr = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (c[:, 0] - a[:, 0])
        T = torch.where((cr < 0)[:, None], T[:, [0, 2, 1]], T)
        v = P[T]
        w = v[:, [1, 2, 0]]
        self.C = C = len(T)
        self.area = 0.5 * cr.abs()
        self.xc = v.mean(dim=1)
        t = w - v
        self.len = torch.sqrt((t ** 2).sum(-1))
        self.n = torch.stack([t[..., 1], -t[..., 0]], -1) / self.len[..., None]
        self.xf = 0.5 * (v + w)
        self.inr = 2 * self.area / self.len.sum(1)
        e0, e1 = T, T[:, [1, 2, 0]]
        key = (torch.minimum(e0, e1) * (len(P) + 1) + torch.maximum(e0, e1)).reshape(-1)
        srt, order = torch.sort(key, stable=True)
        twin = torch.full_like(key, -1)
        same = torch.nonzero(srt[1:] == srt[:-1])[:, 0]
        i, j = order[same], order[same + 1]
        twin[i], twin[j] = j, i
        self.twin = twin.view(C, 3)
        self.nb = torch.where(self.twin >= 0, self.twin // 3, self.twin)
        self.bnd = self.nb < 0
        self.r = self.xf - self.xc[:, None]
        self.nbs = self.nb.clamp(min=0)
        off = torch.where(self.bnd[..., None], 2 * self.r, self.xc[self.nbs] - self.xc[:, None])
        self.wgt = []
        for d in (0, 1):
            M = off * ((~self.bnd) | (self.n[..., d].abs() > 1e-12))[..., None]
            sxx, sxy, syy = (M[..., 0] ** 2).sum(1), (M[..., 0] * M[..., 1]).sum(1), (M[..., 1] ** 2).sum(1)
            det = (sxx * syy - sxy * sxy)[:, None]
            self.wgt.append((syy[:, None] * M[..., 0] - sxy[:, None] * M[..., 1]) / det if d == 0
                            else (sxx[:, None] * M[..., 1] - sxy[:, None] * M[..., 0]) / det)
        inr_nb = torch.where(self.bnd, self.inr[:, None], self.inr[self.nbs])
        self.inr_f = torch.minimum(self.inr[:, None], inr_nb)

    def _mirror(self, qx, qy):
        nx, ny = self.n[..., 0], self.n[..., 1]
        qn = qx * nx + qy * ny
        return qx - 2 * qn * nx, qy - 2 * qn * ny

    def residual(self, Q):
        b, h, qx, qy = Q
        hi = _hinv(h)
        W = [b, b + h, qx * hi, qy * hi]
        ux, uy = self._mirror(W[2][:, None], W[3][:, None])
        ghost = [b[:, None].expand(-1, 3), (b + h)[:, None].expand(-1, 3), ux, uy]
        phis, grads = [], []
        for w, gh in zip(W, ghost):
            wc = w[:, None]
            wn = torch.where(self.bnd, gh, w[self.nbs])
            bd = torch.where(self.bnd, 2 * gh - wc, wn)
            hi_, lo_ = torch.maximum(w, bd.max(1).values), torch.minimum(w, bd.min(1).values)
            gx, gy = (self.wgt[0] * (wn - wc)).sum(1), (self.wgt[1] * (wn - wc)).sum(1)
            ds = [gx * self.r[:, k, 0] + gy * self.r[:, k, 1] for k in range(3)]
            phis.append(_limit("minmod", ds, hi_ - w, lo_ - w, 0.0))
            grads.append((gx, gy))
        wet = (h >= 1e-3).double()
        phis = [p * wet for p in phis]
        phis = [torch.minimum(p, phis[1]) for p in phis]
        own = [w[:, None] + (p * g[0])[:, None] * self.r[..., 0] + (p * g[1])[:, None] * self.r[..., 1]
               for w, p, g in zip(W, phis, grads)]

        def trace(t):
            hf = torch.maximum(t[1], t[0]) - t[0]
            return t[0], hf, [t[2] * hf, t[3] * hf], [t[2], t[3]]
        tw = self.twin.clamp(min=0)
        mx, my = self._mirror(own[2], own[3])
        out = [own[0], own[1], mx, my]
        oth = [torch.where(self.bnd, m, o.reshape(-1)[tw]) for m, o in zip(out, own)]
        nx, ny = self.n[..., 0], self.n[..., 1]
        A = trace(own)
        Fh, Fq, Dm, _ = _flux(A, trace(oth), (nx, ny), "hll_hr")
        gA = 0.5 * G * (h[:, None] + A[1]) * (A[0] - b[:, None])
        k = self.len / self.area[:, None]
        return torch.stack([torch.zeros_like(h), -(k * Fh).sum(1),
                            -(k * (Fq[0] + (Dm + gA) * nx)).sum(1),
                            -(k * (Fq[1] + (Dm + gA) * ny)).sum(1)])

    def dt(self, Q):
        hi = _hinv(Q[1])[:, None]
        lam = (Q[2][:, None] * hi * self.n[..., 0] + Q[3][:, None] * hi * self.n[..., 1]).abs()
        lam = lam + torch.sqrt(G * Q[1].clamp(min=0))[:, None]
        return float((CFL * 2 * self.inr_f / (2 * lam)).min())

    def arrays(self):
        """The solver's mesh arrays: faces numbered by (owner cell, local
        edge), the lower cell owning a shared face."""
        he = torch.arange(3 * self.C, device="cuda").view(self.C, 3)
        owns = self.bnd | (he < self.twin)
        flat = owns.reshape(-1)
        num = torch.cumsum(flat.long(), 0) - 1
        face = torch.where(flat, num, num[self.twin.reshape(-1).clamp(min=0)]).view(self.C, 3)
        srt = torch.argsort(face, dim=1)
        cell = (he // 3)[owns]
        nb = self.nb[owns]
        bd = nb < 0
        xf = self.xf[owns]
        ra = xf - self.xc[cell]
        rb = torch.where(bd[:, None], ra, xf - self.xc[nb.clamp(min=0)])
        n = self.n[owns]
        by_slot = lambda f: torch.gather(f, 1, srt).t().contiguous()  # noqa: E731
        none = {k: None for k in ("lsq_idx", "cell_face", "face_a", "face_b", "bf_kind")}
        return {**none, "lsq_wx": by_slot(self.wgt[0]), "lsq_wy": by_slot(self.wgt[1]),
                "cf_rx": by_slot(self.r[..., 0]), "cf_ry": by_slot(self.r[..., 1]),
                "cell_inv_area": 1 / self.area, "face_nx": n[:, 0], "face_ny": n[:, 1],
                "face_len": self.len[owns], "face_rax": ra[:, 0], "face_ray": ra[:, 1],
                "face_rbx": rb[:, 0], "face_rby": rb[:, 1], "face_inr": self.inr_f[owns],
                "bf_nx": n[bd, 0], "bf_ny": n[bd, 1]}


def _exact_tri(case, seed):
    P, T = _lattice(case["side"], seed)
    m = _Tri(P, T)
    Q = _tri_state(P, T, seed).to(_dtype(case)).double()
    for _ in range(case["steps"]):
        dt = m.dt(Q)
        Q1 = Q + dt * m.residual(Q)
        Qn = 0.5 * (Q + Q1 + dt * m.residual(Q1))
        Q = _friction(Qn, Q[1], dt, case["manning"], True)
    return Q


def _exact_ensemble(case, seed):
    sides, manning, heights = _ens_sides(case, seed)
    out = []
    for i, (n, mn, ht) in enumerate(zip(sides.tolist(), manning.tolist(), heights.tolist())):
        g = _Grid(n, n, 1.0 / n, 1.0 / n, _bc("wall"), "eta", "hll_hr", case["limiter"], 2)
        Q = _ens_state(n, seed + 1 + i, ht).to(_dtype(case)).double().view(4, n, n)
        for _ in range(case["steps"]):
            Q = g.step(Q, g.dt(Q), mn)
        out.append(Q.reshape(-1))
    return torch.cat(out)


def _solve_poisson(cx, cy, f, dx):
    """Diagonally preconditioned conjugate gradients to 1e-13."""
    d = cx[1:] + cx[:-1] + cy[:, 1:] + cy[:, :-1]
    d[0] += cx[0]
    d[-1] += cx[-1]
    d[:, 0] += cy[:, 0]
    d[:, -1] += cy[:, -1]
    dinv = dx * dx / d
    x = torch.zeros_like(f)
    r = f.clone()
    z = dinv * r
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-13 * float(f.norm())
    for it in range(40000):
        q = _poisson(cx, cy, p, dx)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 100 == 99 and float(r.norm()) <= stop:
            break
        z = dinv * r
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_chorin(case, seed):
    nx, ny = case["nx"], case["ny"]
    Q, dx = _chorin_state(case, seed)
    Q = Q.double().view(4, nx, ny)
    dt = 0.2 * dx / 5.0
    g = _Grid(nx, ny, dx, dx, _bc("wall"), "eta", "hll_hr", "minmod", 2)

    def stage(Q):
        Q = Q + dt * g.residual(Q)
        cx, cy = _faces(Q[1], ())
        fx, fy = torch.zeros_like(cx), torch.zeros_like(cy)
        fx[1:-1] = 0.5 * (Q[2][:-1] + Q[2][1:])
        fy[:, 1:-1] = 0.5 * (Q[3][:, :-1] + Q[3][:, 1:])
        f = -((fx[1:] - fx[:-1]) + (fy[:, 1:] - fy[:, :-1])) / (dx * dt)
        p = _solve_poisson(cx, cy, f, dx)
        px = torch.cat([-p[:1], p, -p[-1:]], dim=0)
        py = torch.cat([-p[:, :1], p, -p[:, -1:]], dim=1)
        wx, wy = cx * (px[1:] - px[:-1]) / dx, cy * (py[:, 1:] - py[:, :-1]) / dx
        return torch.stack([Q[0], Q[1], Q[2] - 0.5 * dt * (wx[1:] + wx[:-1]),
                            Q[3] - 0.5 * dt * (wy[:, 1:] + wy[:, :-1])])
    t = 0.0
    for _ in range(case["steps"]):
        Q = stage(Q) if case["time_order"] == 1 else 0.5 * (Q + stage(stage(Q)))
        t += dt
    return Q.view(4, -1), t


def _exact_net(ws, bs, case, r, cx, cy, dx):
    """The network's correction for residuals ``r (B, H, W)``."""
    conv = torch.nn.functional.conv2d
    W, B, i, j = [], [], 0, 0
    for ci, co in _net_shapes(case["c1"], case["c2"]):
        W.append(ws[i:i + co * ci * 9].view(co, ci, 3, 3))
        B.append(bs[j:j + co])
        i, j = i + co * ci * 9, j + co
    s = torch.sqrt((r ** 2).mean(dim=(1, 2), keepdim=True)).clamp(min=1e-30)
    c = 0.25 * (cx[:, :-1] + cx[:, 1:] + cy[:, :, :-1] + cy[:, :, 1:])
    e1 = torch.tanh(conv(torch.stack([r / s, c / 2.0], 1), W[0], B[0], padding=1))
    e2 = torch.tanh(conv(e1, W[1], B[1], padding=1))
    m = torch.tanh(conv(torch.nn.functional.avg_pool2d(e2, 2), W[2], B[2], padding=1))
    m = torch.tanh(conv(m, W[3], B[3], padding=1))
    up = torch.repeat_interleave(torch.repeat_interleave(m, 2, 2), 2, 3)
    o = torch.tanh(conv(torch.cat([up, e2], 1), W[4], B[4], padding=1))
    return s * dx * dx / c * conv(o, W[5], B[5], padding=1)[:, 0]


def exact(case, seed):
    k = case["kind"]
    if k in ("solve", "march", "step"):
        return _exact_flow(case, seed)
    if k == "ensemble":
        return _exact_ensemble(case, seed)
    if k == "tri":
        return _exact_tri(case, seed)
    if k == "trimesh":
        return _Tri(*_lattice(case["side"], seed)).arrays()
    if k == "chorin":
        return _exact_chorin(case, seed)
    w, b = (t.double().cuda() for t in _net(case, seed))
    if k == "smoother":
        nx, ny = case["nx"], case["ny"]
        f, x, cx, cy, dx = _grid_residual(case, seed)
        f, x = f.double().view(1, nx, ny), x.double().view(1, nx, ny)
        cx, cy = cx.double().view(1, nx + 1, ny), cy.double().view(1, nx, ny + 1)
        r = f - _poisson(cx, cy, x, dx)
        return (x + _exact_net(w, b, case, r, cx, cy, dx)).reshape(-1)
    r, cx, cy, e, dx = _patches(case, seed)
    r, cx, cy, e = (t.double() for t in (r, cx, cy, e))
    w.requires_grad_(True)
    b.requires_grad_(True)
    y = _exact_net(w, b, case, r, cx, cy, dx)
    if case["energy"]:
        num = ((e - y) * _poisson(cx, cy, e - y, dx)).sum(dim=(1, 2))
        den = (e * _poisson(cx, cy, e, dx)).sum(dim=(1, 2))
    else:
        num = ((r - _poisson(cx, cy, y, dx)) ** 2).sum(dim=(1, 2))
        den = (r ** 2).sum(dim=(1, 2))
    loss = (num / den).mean()
    gw, gb = torch.autograd.grad(loss, (w, b))
    return loss.detach().reshape(1), gw, gb
