"""The work that programs have this package do, as cases that can be timed and compared.

Every case is a call that a program makes through the public entry points, on fields as they
look in the middle of a run (smoke blobs, a swirling wall-bounded velocity, sources that
inject every step), at the sizes of the package's own configurations, tests and benchmark or
at plain sizes between them. ``listed`` names them, ``draw`` gives more of the same ranges,
``prepare`` makes what the program holds before the call, ``run`` is one call, ``exact`` is
the same call in 64 bits written in plain torch.
"""
import importlib
import math
import random

import torch

sg = importlib.import_module("python-game-engine_b200")
adjoint = importlib.import_module("python-game-engine_b200.adjoint")
batch = importlib.import_module("python-game-engine_b200.batch")
ops = importlib.import_module("python-game-engine_b200.operators")
scenes = importlib.import_module("python-game-engine_b200.scenes")

F64 = torch.float64
BATCH_SIZES = (64, 96, 128, 192, 256)
DISSIPATION = 0.999


# ---------------------------------------------------------------- the cases
def _substep(H, W, dtype, method, **more):
    case = {"kind": "substep", "H": H, "W": W, "dtype": dtype, "method": method, "iterations": 0, "omega": 0.0,
            "tol": 0.0, "precision": "", "coarsest": 0, "smoother": "", "levels": 0, "arithmetic": "reference",
            "source": "plume", "obstacles": False}
    case.update(more)
    return case


def listed():
    cases = {
        # a small interactive window: the default solver of the default configuration, one
        # emitter of smoke and heat, one frame through update()
        "frame_75x50": _substep(50, 75, "float32", "jacobi", iterations=40, source="emitter"),
        # the 128^2 plume configuration: 100 Jacobi sweeps, float64
        "jacobi_128_f64": _substep(128, 128, "float64", "jacobi", iterations=100),
        # an ordinary preview in float32 with the same solver at its default 40 sweeps
        "jacobi_600x800": _substep(600, 800, "float32", "jacobi", iterations=40),
        # the lexicographic Gauss-Seidel solver at its default 40 sweeps, odd sizes
        "gauss_seidel_97x161": _substep(97, 161, "float32", "gauss_seidel", iterations=40),
        # fixed red-black SOR sweeps (omega 1.9, 100 of them) around solid obstacles, ragged
        "sor_obstacles_389x514": _substep(389, 514, "float32", "rb_sor_gauss_seidel", iterations=100, omega=1.9,
                                          obstacles=True),
        # the 512^2 plume with red-black SOR to 1e-6, float64
        "sor_to_1e-6_512_f64": _substep(512, 512, "float64", "rb_sor_tolerance", omega=1.9, tol=1e-6,
                                        precision="native"),
        # the original V-cycle (7 levels, red-black smoother, two cycles) at 512^2
        "vcycles_512": _substep(512, 512, "float32", "multigrid", smoother="rb_sor_gauss_seidel", levels=7,
                                iterations=2),
        # the 512^2 plume with the convergent multigrid to 1e-6, float64, 8^2 coarsest level
        "multigrid_512_f64": _substep(512, 512, "float64", "geometric_multigrid", tol=1e-6, precision="fp64",
                                      coarsest=8),
        # a program's own projection of a velocity field around obstacles, ragged size
        "project_obstacles_421x300": {"kind": "project", "H": 421, "W": 300, "dtype": "float32", "tol": 1e-6,
                                      "precision": "mixed"},
        # the largest single scene: 2048^2, mixed precision to 1e-8, float32 operators
        "multigrid_2048_mixed": _substep(2048, 2048, "float32", "geometric_multigrid", tol=1e-8, precision="mixed",
                                         coarsest=128, arithmetic="float32"),
        # many independent scenes of uneven sizes stepped together
        "batch_256": {"kind": "batch", "scenes": 256, "mix": 1000},
        # inverse problem: loss and gradient of the control through 16 steps, forward and back
        "gradient_256": {"kind": "gradient", "n": 256, "steps": 16},
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "jacobi", "gauss_seidel", "sor", "sor_tol", "vcycles", "multigrid", "project",
                       "large", "batch", "gradient"))
    dtype = rng.choice(("float32", "float64"))

    def grid(lo, hi):
        h = _log(rng, lo, hi)
        return h, max(lo, min(hi, int(h * rng.uniform(0.7, 1.4))))

    if kind == "frame":
        H, W = grid(24, 200)
        return _substep(H, W, "float32", "jacobi", iterations=40, source="emitter")
    if kind == "jacobi":
        H, W = grid(64, 1100)
        return _substep(H, W, dtype, "jacobi", iterations=rng.choice((40, 50, 100)),
                        obstacles=rng.random() < 0.25)
    if kind == "gauss_seidel":
        H, W = grid(32, 180)
        return _substep(H, W, dtype, "gauss_seidel", iterations=rng.choice((20, 40)), obstacles=rng.random() < 0.25)
    if kind == "sor":
        H, W = grid(48, 1100)
        return _substep(H, W, dtype, "rb_sor_gauss_seidel", iterations=rng.choice((40, 100)),
                        omega=rng.choice((0.0, 1.7, 1.9)), obstacles=rng.random() < 0.4)
    if kind == "sor_tol":
        H, W = grid(64, 340)
        return _substep(H, W, dtype, "rb_sor_tolerance", omega=1.9, tol=1e-6,
                        precision="native" if dtype == "float64" else "mixed")
    if kind == "vcycles":
        levels = rng.choice((4, 5, 6))
        H, W = (2 ** (levels - 1) * max(2, v // 2 ** (levels - 1)) for v in grid(96, 1024))
        return _substep(H, W, dtype, "multigrid", smoother=rng.choice(("jacobi", "rb_sor_gauss_seidel")),
                        levels=levels, iterations=2)
    if kind == "multigrid":
        H, W = grid(64, 1024)
        return _substep(H, W, dtype, "geometric_multigrid", tol=rng.choice((1e-6, 1e-8)),
                        precision="fp64" if dtype == "float64" else "mixed", coarsest=8)
    if kind == "project":
        H, W = grid(64, 700)
        return {"kind": "project", "H": H, "W": W, "dtype": dtype, "tol": 1e-6,
                "precision": "fp64" if dtype == "float64" else "mixed"}
    if kind == "large":
        H, W = (128 * rng.randint(8, 16) for _ in range(2))
        return _substep(H, W, dtype, "geometric_multigrid", tol=1e-8, coarsest=128,
                        precision="fp64" if dtype == "float64" else "mixed",
                        arithmetic="reference" if dtype == "float64" else rng.choice(("reference", "float32")))
    if kind == "batch":
        return {"kind": "batch", "scenes": _log(rng, 12, 256), "mix": rng.randint(0, 10 ** 6)}
    return {"kind": "gradient", "n": 4 * rng.randint(16, 64), "steps": rng.choice((4, 6, 8, 12, 16))}


def work(case):
    """Each field read once and written once; the sweeps a fixed-count solver is asked for."""
    if case["kind"] == "batch":
        cells, size, passes, flops = sum(n * n for n in _sizes(case)), 4, 9, 120
    elif case["kind"] == "gradient":
        # every step forward and back: state and control in, their adjoints out
        cells, size, passes, flops = case["n"] ** 2 * case["steps"], 4, 14, 400
    else:
        cells, size = case["H"] * case["W"], 8 if case["dtype"] == "float64" else 4
        passes, flops = (5, 20) if case["kind"] == "project" else (9, 120)
        if case["kind"] == "substep" and case["method"] != "multigrid":
            flops += 8 * case["iterations"]
        elif case["kind"] == "substep":  # two V(2,2) cycles
            flops += 2 * 50
    return {"bytes": passes * size * cells, "flops": flops * cells}


# ---------------------------------------------------------------- inputs
def _dtype(case):
    return torch.float64 if case["dtype"] == "float64" else torch.float32


def _axes(rows, cols, dev):
    return torch.meshgrid(torch.arange(rows, dtype=F64, device=dev), torch.arange(cols, dtype=F64, device=dev),
                          indexing="ij")


def _fields(H, W, rng, dev):
    """Density and velocity in the middle of a run, in float64: smoke blobs, and the curl of a
    wall-bounded stream function (speed about 1, zero on the faces next to the walls)."""
    h = 1.0 / max(H, W)
    j, i = _axes(H, W, dev)
    d = torch.zeros((H, W), dtype=F64, device=dev)
    for _ in range(5):
        cx, cy, r = rng.uniform(0.15, 0.85) * W, rng.uniform(0.15, 0.85) * H, rng.uniform(0.04, 0.12) * min(H, W)
        d += rng.uniform(0.4, 1.0) * torch.exp(-((i + 0.5 - cx) ** 2 + (j + 0.5 - cy) ** 2) / (2.0 * r * r))
    d.clamp_(max=1.0)
    j, i = _axes(H + 1, W + 1, dev)
    psi = torch.zeros_like(j)
    for _ in range(6):
        m, n = rng.randint(1, 5), rng.randint(1, 5)
        psi += rng.uniform(-1.0, 1.0) / (m + n) * torch.sin(math.pi * m * i / W) * torch.sin(math.pi * n * j / H)
    u, v = (psi[1:] - psi[:-1]) / h, -(psi[:, 1:] - psi[:, :-1]) / h
    speed = float(torch.maximum(u.abs().max(), v.abs().max()))
    a = rng.uniform(0.7, 1.2) / speed
    ou, ov = _inner_faces(H, W, _ring(H, W, dev))
    return d, a * u * ou, a * v * ov


def _ring(H, W, dev):
    s = torch.zeros((H, W), dtype=torch.bool, device=dev)
    s[0], s[-1], s[:, 0], s[:, -1] = True, True, True, True
    return s


def _obstacles(H, W, rng, dev):
    """A walled box with three round obstacles."""
    s = _ring(H, W, dev)
    j, i = _axes(H, W, dev)
    for _ in range(3):
        cx, cy, r = rng.uniform(0.2, 0.8) * W, rng.uniform(0.3, 0.8) * H, rng.uniform(0.05, 0.1) * min(H, W)
        s |= (i + 0.5 - cx) ** 2 + (j + 0.5 - cy) ** 2 < r * r
    return s


def _plumes(H, W, rng, count):
    """Rows (x, y, radius, density, inflow speed, noise) in cells, near the bottom."""
    return [[rng.uniform(0.2, 0.8) * W, rng.uniform(0.08, 0.2) * H, rng.uniform(0.03, 0.08) * min(H, W), 1.0,
             rng.uniform(0.5, 1.5), 0.0] for _ in range(count)]


def _emitter(H, W, rng):
    return {"position": (rng.uniform(0.3, 0.7) * W, rng.uniform(0.15, 0.3) * H), "radius": 0.12 * min(H, W),
            "density": 8.0, "temperature": 30.0, "velocity": (rng.uniform(-4.0, 4.0), 20.0)}


def _scene(case, seed, dev):
    """All that a substep starts from, in float64 rounded to the case's type."""
    H, W = case["H"], case["W"]
    rng = random.Random(seed)
    d, u, v = _fields(H, W, rng, dev)
    s = {"h": 1.0 / max(H, W), "solid": None, "emitter": None, "plumes": [], "t": None}
    s["dt"] = 0.5 * s["h"]
    s["d"], s["u"], s["v"] = (x.to(_dtype(case)) for x in (d, u, v))
    if case["kind"] == "project" or case["obstacles"]:
        s["solid"] = _obstacles(H, W, rng, dev)
    if case["kind"] == "substep" and case["source"] == "emitter":
        s["emitter"] = _emitter(H, W, rng)
        s["t"] = (0.5 * d).to(_dtype(case))
    else:
        s["plumes"] = _plumes(H, W, rng, 4 if max(H, W) >= 1024 else 1)
    if case["kind"] == "project":  # sources have just injected: the field is not divergence-free
        s["u"], s["v"] = (x.to(_dtype(case)) for x in _inject(d, u, v, s["plumes"])[1:])
    return s


def _sizes(case):
    rng = random.Random(case["mix"])
    return [rng.choice(BATCH_SIZES) for _ in range(case["scenes"])]


def _batch_scenes(case, seed, dev):
    """(scene, density, u, v) of every member, in float32."""
    rng = random.Random(seed)
    got = []
    for k, n in enumerate(_sizes(case)):
        row = [rng.uniform(0.2, 0.8) * n, rng.uniform(0.08, 0.25) * n, rng.uniform(0.04, 0.16) * n, 1.0, 1.0, 0.0]
        sc = scenes.Scene(f"scene_{k}", n, n, 1, -rng.uniform(0.5, 2.0), [row], seed=seed)
        got.append((sc, *(x.float() for x in _fields(n, n, rng, dev))))
    return got


def _control(case, seed):
    """Plume row, control force and target blob of an inverse problem."""
    n = case["n"]
    rng = random.Random(seed)
    plume = [rng.uniform(0.3, 0.7) * n, 0.12 * n, 12.0 * n / 256, 1.0, 1.0, 0.0]
    gen = torch.Generator().manual_seed(seed)
    force = (0.01 * torch.randn((case["steps"], 2, n, n), generator=gen)).cuda()
    cx, cy, sigma = plume[0] + rng.uniform(-0.05, 0.05) * n, 0.2 * n, 20.0 * n / 256
    j, i = _axes(n, n, "cuda")
    target = torch.exp(-((i + 0.5 - cx) ** 2 + (j + 0.5 - cy) ** 2) / (2.0 * sigma * sigma)).float()
    return plume, force, target


# ---------------------------------------------------------------- one pass
def _params(case):
    m = case["method"]
    if m == "jacobi":
        return sg.JacobiParams(iterations=case["iterations"])
    if m == "gauss_seidel":
        return sg.GaussSeidelParams(iterations=case["iterations"])
    if m == "rb_sor_gauss_seidel":
        return sg.SORParams(iterations=case["iterations"], omega=case["omega"])
    if m == "rb_sor_tolerance":
        return sg.SORToleranceParams(omega=case["omega"], tol=case["tol"], precision=case["precision"])
    if m == "multigrid":
        return sg.MultigridParams(smoother_type=case["smoother"], num_levels=case["levels"],
                                  smoother_iterations=case["iterations"])
    return sg.GeometricMultigridParams(tol=case["tol"], precision=case["precision"], coarsest=case["coarsest"])


def _prepare_substep(case, seed):
    s = _scene(case, seed, "cuda")
    H, W = case["H"], case["W"]
    cfg = sg.SimulationConfig(grid=sg.GridConfig(size=(W, H), cell_size=s["h"]),
                              pressure_solver=sg.PressureSolverConfig(method=case["method"], params=_params(case)))
    sim = sg.SmokeSimulation2D(cfg, dtype=_dtype(case), seed=seed)
    sim.dt, sim.gravity = s["dt"], -1.0
    sim.advection_arithmetic = sim.operator_arithmetic = case["arithmetic"]
    sim.density.copy_(s["d"])
    sim.velocity_u.copy_(s["u"])
    sim.velocity_v.copy_(s["v"])
    if s["emitter"]:
        e = s["emitter"]
        sim.temperature.copy_(s["t"])
        sim.add_emitter(sg.Emitter2D(e["position"], e["radius"], density_value=e["density"],
                                     temperature_value=e["temperature"], velocity_value=e["velocity"]))
    else:
        sim.set_plumes([sg.PlumeSource(*row) for row in s["plumes"]])
    if s["solid"] is not None:
        sim.set_solid_mask(s["solid"])
    return {"sim": sim, "case": case}


def _run_substep(state):
    sim, case = state["sim"], state["case"]
    if case["source"] == "emitter":
        sim.update(sim.dt)
    else:
        sim.substep(sim.dt)
    out = {"density": sim.density, "u": sim.velocity_u, "v": sim.velocity_v, "pressure": sim.pressure}
    if case["source"] == "emitter":
        out["temperature"] = sim.temperature
    if case["iterations"]:  # after a solve to a tolerance these two hold rounding remainders only
        out["divergence"], out["residual"] = sim.divergence, sim.pressure_residual
    return out


def _prepare_project(case, seed):
    s = _scene(case, seed, "cuda")
    fmu, fmv, fluid = ops.build_masks(s["solid"])
    z = torch.zeros_like(s["d"])
    return {"case": case, "s": s, "fmu": fmu, "fmv": fmv, "solver": sg.GeometricMultigridSolver(), "div": z,
            "p": torch.zeros_like(z), "u": torch.empty_like(s["u"]), "v": torch.empty_like(s["v"])}


def _run_project(t):
    s, case = t["s"], t["case"]
    ops.compute_divergence(s["u"], s["v"], t["div"], t["fmu"], t["fmv"], s["h"])
    t["p"].zero_()
    t["solver"](t["p"], t["div"], t["fmu"], t["fmv"], 1.0, s["h"], s["dt"], tol=case["tol"],
                precision=case["precision"], zero_initial_guess=True)
    t["u"].copy_(s["u"])
    t["v"].copy_(s["v"])
    ops.project(t["u"], t["v"], t["p"], t["fmu"], t["fmv"], s["solid"], 1.0, s["h"], s["dt"])
    return {"u": t["u"], "v": t["v"], "pressure": t["p"], "divergence": t["div"]}


def _pools(b):
    """Density, u, v and pressure of all scenes, one after another (views of the arena)."""
    first, last = b.fields(0), b.fields(len(b.scenes) - 1)
    whole = b.workspace[:b.bytes // 4 * 4].view(torch.float32)
    out = []
    for x, y in zip(first, last):
        lo = x.storage_offset()
        out.append(whole[lo:y.storage_offset() + y.numel()])
    return out


def _prepare_batch(case, seed):
    members = _batch_scenes(case, seed, "cuda")
    b = batch.BatchedSmoke([m[0] for m in members], tol=1e-6, seed=seed)
    b.configure(sweeps=2, cycle="V")
    for k, m in enumerate(members):
        for dst, src in zip(b.fields(k), m[1:]):
            dst.copy_(src)
    return {"batch": b}


def _run_batch(state):
    state["batch"].step()
    return dict(zip(("density", "u", "v", "pressure"), _pools(state["batch"])))


def _prepare_gradient(case, seed):
    plume, force, target = _control(case, seed)
    n = case["n"]
    model = adjoint.ControlledSmoke(n, n, 1.0 / n, 0.5 / n, gravity=-1.0, plumes=[plume], seed=seed)
    return {"model": model, "force": force, "target": target}


def _run_gradient(t):
    loss, grad = adjoint.loss_and_grad(t["model"], t["force"], t["target"])
    return {"loss": loss, "grad": grad}


def prepare(case, seed):
    return {"substep": _prepare_substep, "project": _prepare_project, "batch": _prepare_batch,
            "gradient": _prepare_gradient}[case["kind"]](case, seed)


def run(state):
    if "sim" in state:
        return _run_substep(state)
    if "batch" in state:
        return _run_batch(state)
    return _run_gradient(state) if "model" in state else _run_project(state)


# ---------------------------------------------------------------- the same in 64 bits
def _sample(f, x, y):
    """Clamped bilinear sample at (x, y) in index space."""
    rows, cols = f.shape
    x0, x1 = torch.floor(x).clamp(0, cols - 1), torch.ceil(x).clamp(0, cols - 1)
    y0, y1 = torch.floor(y).clamp(0, rows - 1), torch.ceil(y).clamp(0, rows - 1)
    tx, ty = x - x0, y - y0
    x0, x1, y0, y1 = (k.long() for k in (x0, x1, y0, y1))
    a = f[y0, x0] + (f[y0, x1] - f[y0, x0]) * tx
    b = f[y1, x0] + (f[y1, x1] - f[y1, x0]) * tx
    return a + (b - a) * ty


def _faces(H, W, solid, dev):
    """Open faces (u, v) and fluid cells; without a plane every interior face is open."""
    mu = torch.zeros((H, W + 1), dtype=torch.bool, device=dev)
    mv = torch.zeros((H + 1, W), dtype=torch.bool, device=dev)
    s = torch.zeros((H, W), dtype=torch.bool, device=dev) if solid is None else solid
    mu[:, 1:-1] = ~(s[:, 1:] | s[:, :-1])
    mv[1:-1] = ~(s[1:] | s[:-1])
    return mu, mv, mu[:, 1:] | mu[:, :-1] | mv[1:] | mv[:-1]


def _inner_faces(H, W, solid):
    """1 where neither neighbouring cell is solid and the face is not the domain's edge."""
    mu, mv, _ = _faces(H, W, solid, solid.device)
    return mu.to(F64), mv.to(F64)


def _inject(d, u, v, plumes):
    H, W = d.shape
    cj, ci = _axes(H + 1, W + 1, d.device)
    for cx, cy, r, dens, speed, _noise in plumes:
        hit = ((ci + 0.5 - cx) ** 2 + (cj + 0.5 - cy) ** 2 < r * r)[:H, :W]
        d = torch.where(hit, torch.full_like(d, dens), d)
        hit = ((ci + 0.5 - cx) ** 2 + (cj - cy) ** 2 < r * r)[:, :W]
        v = torch.where(hit, torch.full_like(v, speed), v)
        hit = ((ci - cx) ** 2 + (cj + 0.5 - cy) ** 2 < r * r)[:H]
        u = torch.where(hit, torch.zeros_like(u), u)
    return d, u, v


def _emit(f, value, e, dt):
    j, i = _axes(*f.shape, f.device)
    dist = torch.sqrt((i - e["position"][0]) ** 2 + (j - e["position"][1]) ** 2)
    return f + torch.where(dist < e["radius"], value * (1.0 - dist / e["radius"]) * dt, torch.zeros_like(dist))


def _mean_rows(x):
    return torch.cat([x[:1], 0.5 * (x[:-1] + x[1:]), x[-1:]], 0)


def _buoyancy(d, t, gravity, coefficient):
    """Force on the v faces: density on faces 0 .. H-1 (its own value on the first and the last
    of them, the mean of two cells between), heat on all of them."""
    dd = _mean_rows(d)
    dd[-2], dd[-1] = d[-1], 0.0
    f = -dd * gravity
    return f if t is None else f - coefficient * _mean_rows(t)


def _advect_velocity(u, v, k, mu, mv):
    H, W = u.shape[0], v.shape[1]
    j, i = _axes(H, W + 1, u.device)
    x, y = i - u * k, j + 0.5 - _sample(v, i - 0.5, j + 0.5) * k
    u2 = _sample(u, x, y - 0.5) * mu
    j, i = _axes(H + 1, W, u.device)
    x, y = i + 0.5 - _sample(u, i + 0.5, j - 0.5) * k, j - v * k
    return u2, _sample(v, x - 0.5, y) * mv


def _advect_cells(f, u, v, k, fluid):
    j, i = _axes(*f.shape, f.device)
    x, y = i - _sample(u, i + 0.5, j) * k, j - _sample(v, i, j + 0.5) * k
    return _sample(f, x, y) * fluid


def _divergence(u, v, mu, mv, h):
    u, v = u * mu, v * mv
    return ((u[:, 1:] - u[:, :-1]) + (v[1:] - v[:-1])) / h


def _neighbours(p, mu, mv):
    """Sum of the four neighbours, the cell itself across a closed face."""
    l, r, d, up = (torch.empty_like(p) for _ in range(4))
    l[:, 1:], l[:, 0] = p[:, :-1], p[:, 0]
    r[:, :-1], r[:, -1] = p[:, 1:], p[:, -1]
    d[1:], d[0] = p[:-1], p[0]
    up[:-1], up[-1] = p[1:], p[-1]
    return (torch.where(mu[:, :-1], l, p) + torch.where(mu[:, 1:], r, p) + torch.where(mv[:-1], d, p)
            + torch.where(mv[1:], up, p))


def _jacobi(p, b, mu, mv, fluid, count):
    for _ in range(count):
        p = torch.where(fluid, 0.25 * (_neighbours(p, mu, mv) + b), p)
    return p


def _red_black(p, b, mu, mv, fluid, count, omega):
    H, W = p.shape
    if not 0.0 < omega <= 2.0:
        omega = min(2.0 / (1.0 + math.sin(math.pi / max(H, W))), 1.95)
    j, i = _axes(H, W, p.device)
    red = ((i + j) % 2 == 0) & fluid
    black = fluid & ~red
    for _ in range(count):
        for mask in (red, black):
            p = torch.where(mask, (1.0 - omega) * p + omega * 0.25 * (_neighbours(p, mu, mv) + b), p)
    return p


def _gauss_seidel(p, b, mu, mv, fluid, count):
    """Rows upward, each from the left, as anti-diagonals; a padded copy holds the grid."""
    H, W = p.shape
    W2 = W + 2
    q = torch.zeros((H + 2, W2), dtype=F64, device=p.device)
    q[1:-1, 1:-1] = p
    q = q.reshape(-1)
    open_ = [m.to(F64).reshape(-1) for m in (mu[:, :-1], mu[:, 1:], mv[:-1], mv[1:])]
    closed = 4.0 - sum(open_)
    diagonals = []
    for s in range(H + W - 1):
        j = torch.arange(max(0, s - W + 1), min(s, H - 1) + 1, device=p.device)
        j = j[fluid[j, s - j]]
        g, k = j * W + (s - j), (j + 1) * W2 + (s - j) + 1
        near = torch.stack([k - 1, k + 1, k - W2, k + W2])
        diagonals.append((k, near, torch.stack([o[g] for o in open_]), closed[g], b.reshape(-1)[g]))
    for _ in range(count):
        for k, near, o, c, bb in diagonals:
            q[k] = 0.25 * ((q[near] * o).sum(0) + c * q[k] + bb)
    return q.reshape(H + 2, W2)[1:-1, 1:-1].clone()


def _vcycles(b0, case, h, dt, solid, dev):
    """Two V-cycles of the original method from p = 0 (b0: divergence)."""
    sizes = [tuple(b0.shape)]
    solids = [~_faces(*sizes[0], solid, dev)[2]]
    while len(sizes) < case["levels"] and sizes[-1][0] % 2 == 0 and sizes[-1][1] % 2 == 0:
        s = solids[-1]
        solids.append(s[::2, ::2] | s[1::2, ::2] | s[::2, 1::2] | s[1::2, 1::2])
        sizes.append(tuple(solids[-1].shape))
    masks = [_faces(*sizes[0], solid, dev)] + [_faces(*z, s, dev) for z, s in zip(sizes[1:], solids[1:])]

    def smooth(k, p, rhs, count):
        b = -(h * 2 ** k) ** 2 / dt * rhs
        return (_jacobi(p, b, *masks[k], count) if case["smoother"] == "jacobi"
                else _red_black(p, b, *masks[k], count, 0.0))

    def cycle(k, p, rhs):
        if k == len(sizes) - 1:
            return smooth(k, p, rhs, 30)
        p = smooth(k, p, rhs, case["iterations"])
        mu, mv, fluid = masks[k]
        r = torch.where(fluid, _neighbours(p, mu, mv) - (h * 2 ** k) ** 2 / dt * rhs - 4.0 * p, torch.zeros_like(p))
        H, W = sizes[k]
        f = fluid.to(F64).reshape(H // 2, 2, W // 2, 2)
        total = (r.reshape(H // 2, 2, W // 2, 2) * f).sum((1, 3)) / f.sum((1, 3)).clamp(min=1.0)
        e = cycle(k + 1, torch.zeros_like(total), total / (-(h * 2 ** (k + 1)) ** 2 / dt))
        j, i = _axes(H, W, dev)
        p = p + torch.where(fluid, _sample(e, (i + 0.5) * 0.5 - 0.5, (j + 0.5) * 0.5 - 0.5), torch.zeros_like(p))
        return smooth(k, p, rhs, case["iterations"])

    p = torch.zeros_like(b0)
    for _ in range(2):
        p = cycle(0, p, b0)
    return p


class _BoxSolve(torch.autograd.Function):
    """-(four-neighbour Laplacian with closed walls)^-1 by cosine transforms; its own transpose."""

    @staticmethod
    def forward(ctx, b):
        H, W = b.shape

        def basis(n):
            k = torch.arange(n, dtype=F64, device=b.device)
            c = torch.cos(math.pi / n * (k[None, :] + 0.5) * k[:, None]) * math.sqrt(2.0 / n)
            c[0] /= math.sqrt(2.0)
            return c, 4.0 * torch.sin(math.pi * k / (2 * n)) ** 2

        (cy, ly), (cx, lx) = basis(H), basis(W)
        t = cy @ b @ cx.T
        lam = ly[:, None] + lx[None, :]
        lam[0, 0] = 1.0
        t = t / lam
        t[0, 0] = 0.0
        return cy.T @ t @ cx

    @staticmethod
    def backward(ctx, g):
        return _BoxSolve.apply(g)


def _conjugate_gradients(b, mu, mv, fluid):
    f = fluid.to(F64)
    n = (mu[:, 1:].to(F64) + mu[:, :-1].to(F64) + mv[1:].to(F64) + mv[:-1].to(F64)).clamp(min=1.0)

    def apply(x):
        return (4.0 * x - _neighbours(x, mu, mv)) * f

    x, r = torch.zeros_like(b), b * f
    z = r / n
    s, rz, stop = z, (r * z).sum(), 1e-26 * float((r * r).sum())
    for k in range(20000):
        a = apply(s)
        step = rz / (s * a).sum()
        x, r = x + step * s, r - step * a
        if k % 50 == 49 and float((r * r).sum()) <= stop:
            break
        z = r / n
        rz, old = (r * z).sum(), rz
        s = z + rz / old * s
    return x


def _pressure(case, div, masks, h, dt, solid):
    """The pressure that the case's solver is asked for, or (for a tolerance) the solution."""
    b = -h * h / dt * div
    m, count = case.get("method"), case.get("iterations")
    if m == "jacobi":
        return _jacobi(torch.zeros_like(b), b, *masks, count)
    if m == "rb_sor_gauss_seidel":
        return _red_black(torch.zeros_like(b), b, *masks, count, case["omega"])
    if m == "gauss_seidel":
        return _gauss_seidel(torch.zeros_like(b), b, *masks, count)
    if m == "multigrid":
        return _vcycles(div, case, h, dt, solid, div.device)
    return _BoxSolve.apply(b) if solid is None else _conjugate_gradients(b, *masks)


def _gradient_step(u, v, p, keep_u, keep_v, mu, mv, scale):
    gu, gv = torch.zeros_like(u), torch.zeros_like(v)
    gu[:, 1:-1] = p[:, 1:] - p[:, :-1]
    gv[1:-1] = p[1:] - p[:-1]
    return (u - scale * gu) * keep_u * mu, (v - scale * gv) * keep_v * mv


def _exact_substep(case, seed):
    H, W = case["H"], case["W"]
    s = _scene(case, seed, "cuda")
    d, u, v = (s[k].to(F64) for k in "duv")
    t = None if s["t"] is None else s["t"].to(F64)
    h, dt, e = s["h"], s["dt"], s["emitter"]
    if e:
        d, t = _emit(d, e["density"], e, dt), _emit(t, e["temperature"], e, dt)
        u, v = _emit(u, e["velocity"][0], e, dt), _emit(v, e["velocity"][1], e, dt)
    d, u, v = _inject(d, u, v, s["plumes"])
    masks = mu, mv, fluid = _faces(H, W, s["solid"], d.device)
    v = v + dt * _buoyancy(d, t, -1.0, 5.0)
    u, v = _advect_velocity(u, v, dt / h, mu, mv)
    d = DISSIPATION * _advect_cells(d, u, v, dt / h, fluid)
    if t is not None:
        t = _advect_cells(t, u, v, dt / h, fluid) * math.exp(-0.5 * dt)
    p = _pressure(case, _divergence(u, v, mu, mv, h), masks, h, dt, s["solid"])
    keep = _inner_faces(H, W, s["solid"] if s["solid"] is not None else _ring(H, W, d.device))
    u, v = _gradient_step(u, v, p, *keep, mu, mv, dt / h)
    # a solve to a tolerance leaves the pressure's constant open: there is no exact value
    out = {"density": d, "u": u, "v": v, "pressure": p if case["iterations"] else None}
    if t is not None:
        out["temperature"] = t
    if case["iterations"]:
        out["divergence"] = _divergence(u, v, mu, mv, h)
        out["residual"] = (_neighbours(p, mu, mv) - h * h / dt * out["divergence"] - 4.0 * p) * fluid
    return out


def _exact_project(case, seed):
    H, W = case["H"], case["W"]
    s = _scene(case, seed, "cuda")
    u, v = s["u"].to(F64), s["v"].to(F64)
    masks = mu, mv, _ = _faces(H, W, s["solid"], u.device)
    div = _divergence(u, v, mu, mv, s["h"])
    p = _pressure(case, div, masks, s["h"], s["dt"], s["solid"])
    u, v = _gradient_step(u, v, p, *_inner_faces(H, W, s["solid"]), mu, mv, s["dt"] / s["h"])
    return {"u": u, "v": v, "pressure": None, "divergence": div}


def _exact_batch(case, seed):
    pools = [[], [], []]
    for sc, d, u, v in _batch_scenes(case, seed, "cuda"):
        n, h, dt = sc.W, sc.cell_size, sc.dt
        d, u, v = _inject(d.to(F64), u.to(F64), v.to(F64), sc.plumes)
        mu, mv, fluid = _faces(n, n, None, d.device)
        v = v + dt * _buoyancy(d, None, sc.gravity, 0.0)
        u, v = _advect_velocity(u, v, dt / h, mu, mv)
        d = DISSIPATION * _advect_cells(d, u, v, dt / h, fluid)
        p = _BoxSolve.apply(-h * h / dt * _divergence(u, v, mu, mv, h))
        u, v = _gradient_step(u, v, p, *_inner_faces(n, n, _ring(n, n, d.device)), mu, mv, dt / h)
        for pool, x in zip(pools, (d, u, v)):
            pool.append(x.reshape(-1))
    d, u, v = (torch.cat(x) for x in pools)
    return {"density": d, "u": u, "v": v, "pressure": None}


def _exact_gradient(case, seed):
    n = case["n"]
    plume, force, target = _control(case, seed)
    h, dt = 1.0 / n, 0.5 / n
    f = force.to(F64).requires_grad_(True)
    d = torch.zeros((n, n), dtype=F64, device=f.device)
    u, v = torch.zeros((n, n + 1), dtype=F64, device=f.device), torch.zeros((n + 1, n), dtype=F64, device=f.device)
    mu, mv, fluid = _faces(n, n, None, d.device)
    keep = _inner_faces(n, n, _ring(n, n, d.device))
    for k in range(case["steps"]):
        d, u, v = _inject(d, u, v, [plume])
        v = v + dt * _buoyancy(d, None, -1.0, 0.0)
        u = torch.cat([u[:, :n] + dt * f[k, 0], u[:, n:]], 1)
        v = torch.cat([v[:n] + dt * f[k, 1], v[n:]], 0)
        u, v = _advect_velocity(u, v, dt / h, mu, mv)
        d = DISSIPATION * _advect_cells(d, u, v, dt / h, fluid)
        p = _BoxSolve.apply(-h * h / dt * _divergence(u, v, mu, mv, h))
        u, v = _gradient_step(u, v, p, *keep, mu, mv, dt / h)
    loss = ((d - target.to(F64)) ** 2).sum()
    (grad,) = torch.autograd.grad(loss, f)
    return {"loss": float(loss.detach()), "grad": grad}


def exact(case, seed):
    return {"substep": _exact_substep, "project": _exact_project, "batch": _exact_batch,
            "gradient": _exact_gradient}[case["kind"]](case, seed)
