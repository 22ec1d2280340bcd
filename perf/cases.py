"""The work a program has this library do, as cases that can be timed.

Four kinds, each through the package's public entry points:

  operator   Simulator.apply_operator: four products in a row, as a caller's
             own iteration makes them (a polynomial smoother, a power method),
             the result mapped back to the caller's particle order
  run        Simulator.makeReady + advance + get: a simulation from the
             caller's host arrays, positions read back once per frame
  batch      Batch.makeReady + advance + get: many bodies stepped together
  network    mlp_predict / mlp_loss_grad: the learned warm start's network

Bodies are jittered simple-cubic lattices, as the reference's Scene fills
them (src/examples/scene.cpp:33-135), or scattered far enough from the sites
that they are no lattice any more.  Every input comes from the seed alone.
"""
import importlib
import math

import numpy as np
import torch

pd = importlib.import_module("sci-solver_peridynamic_gb300")

F = np.float64
PRODUCTS = 4
RIGID_RADIUS, RIGID_SPEED = 0.1, 10.0
ELLIPSOID = (0.5, 0.35, 0.3)


def listed():
    return [
        # products of a small body: launch latency and host calls count
        dict(name="operator_4k_block", kind="operator", shape="block", n=4096, coeff=5.0, jitter=0.05, fp64=False),
        # the benchmark's body: products at the size the metric names
        dict(name="operator_1m_ellipsoid", kind="operator", shape="ellipsoid", n=1_000_000, coeff=5.0, jitter=0.05,
             fp64=False),
        # a body that is no lattice fill: per-bond gathers
        dict(name="operator_200k_scattered", kind="operator", shape="ball", n=200_000, coeff=5.0, jitter=0.4, fp64=False),
        # the precision study's arithmetic and horizon
        dict(name="operator_100k_fp64", kind="operator", shape="beam", n=100_000, coeff=6.0, jitter=0.05, fp64=True),
        # the smallest simulation, read back every step as a viewer does
        dict(name="run_512_block", kind="run", shape="block", n=512, coeff=5.0, jitter=0.05, fp64=False, guess=0,
             tolerance=1e-8, steps=60, frame=1),
        # the small workload: 16^3 particles, implicit Euler
        dict(name="run_4k_block", kind="run", shape="block", n=4096, coeff=5.0, jitter=0.05, fp64=False, guess=0,
             tolerance=1e-8, steps=60, frame=2),
        # three-point bending with breaking bonds and the adaptive time step
        dict(name="run_50k_beam", kind="run", shape="beam", n=50_000, coeff=6.0, jitter=0.05, fp64=False, guess=0,
             tolerance=1e-6, steps=45, frame=15),
        # the benchmark's workload: impact of a rigid sphere, history-projection guess
        dict(name="run_1m_ellipsoid", kind="run", shape="ellipsoid", n=1_000_000, coeff=5.0, jitter=0.05, fp64=False,
             guess=2, tolerance=1e-6, steps=10, frame=1),
        # everything in 64 bits, with a tight solver
        dict(name="run_15k_fp64", kind="run", shape="block", n=15_000, coeff=5.0, jitter=0.05, fp64=True, guess=0,
             tolerance=1e-12, steps=15, frame=5),
        # many bodies of mixed size, horizon and loading
        dict(name="batch_24", kind="batch", count=24, n=4000, n_most=24_000, tolerance=1e-6, steps=12),
        # inference over the rows of a step, and a training gradient
        dict(name="network_predict_100k", kind="network", rows=100_000, grad=False),
        dict(name="network_gradient_12k", kind="network", rows=12_000, grad=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "operator", "run", "run", "batch", "network"])
    if kind == "operator":
        fp64 = rng.random() < 0.25
        return dict(kind=kind, shape=rng.choice(["block", "ball", "beam", "ellipsoid"]),
                    n=_log_int(rng, 500, 200_000 if fp64 else 1_000_000), coeff=rng.choice([4.0, 5.0, 6.0]),
                    jitter=rng.choice([0.05, 0.1, 0.4]), fp64=fp64)
    if kind == "run":
        fp64 = rng.random() < 0.25
        shape = rng.choice(["block", "ball", "beam", "ellipsoid"])
        steps = rng.randrange(8, 25)
        return dict(kind=kind, shape=shape, n=_log_int(rng, 5000 if shape == "ellipsoid" else 400, 20_000 if fp64 else 250_000),
                    coeff=rng.choice([4.0, 5.0, 6.0]), jitter=0.05, fp64=fp64, guess=rng.choice([0, 0, 2]),
                    tolerance=1e-12 if fp64 else 1e-8 if shape == "block" else 1e-6, steps=steps, frame=rng.randrange(1, steps))
    if kind == "batch":
        n = _log_int(rng, 800, 6000)
        return dict(kind=kind, count=rng.randrange(4, 33), n=n, n_most=n * rng.randrange(1, 5), tolerance=1e-6,
                    steps=rng.randrange(5, 16))
    return dict(kind=kind, rows=_log_int(rng, 100, 200_000), grad=False) if rng.random() < 0.6 else \
        dict(kind=kind, rows=_log_int(rng, 100, 20_000), grad=True)


# ---- bodies -------------------------------------------------------------------------
def _lattice(nx, ny, nz):
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)


def _body(shape, n, coeff, jitter, seed):
    """Sites, positions, activity, velocity and constants (SI units; density 125
    kg/m^3 and a bond stiffness under which the wave speed does not depend on
    the spacing)."""
    rng = np.random.default_rng(seed)
    body = {"coeff": coeff, "sphere": None}
    if shape == "block":                       # clamped base, top layer driven down
        side = max(2, int(round(n ** (1 / 3))))
        g = _lattice(side, side, max(2, int(round(n / side ** 2))))
        h, newmark, dt, s0 = 0.02, False, 1e-4, 0.02
    elif shape == "ball":                      # struck by a rigid sphere half its size
        R = (3 * n / (4 * math.pi)) ** (1 / 3)
        m = int(math.ceil(R)) + 1
        g = _lattice(2 * m + 1, 2 * m + 1, 2 * m + 1) - m
        g = g[(g.astype(F) ** 2).sum(1) <= R * R]
        h, newmark, dt, s0 = 0.02, True, 5e-5, 0.02
    elif shape == "beam":                      # 5:1:1, notched, three-point bending
        h = (1.0 * 0.2 * 0.2 / n) ** (1 / 3)
        g = _lattice(*(max(2, int(round(s / h))) for s in (1.0, 0.2, 0.2)))
        p = (g + 0.5) * h
        keep = ~((np.abs(p[:, 0] - 0.5) < h) & (p[:, 2] < 0.05))
        g, p = g[keep], p[keep]
        newmark, dt, s0 = True, 5e-5, 0.01
    else:                                      # ellipsoid struck by a rigid sphere, as the benchmark
        h = (4 / 3 * math.pi * ELLIPSOID[0] * ELLIPSOID[1] * ELLIPSOID[2] / n) ** (1 / 3)
        dims = [int(math.floor(2 * s / h)) + 1 for s in ELLIPSOID]
        g = _lattice(*dims)
        p = (g - (np.array(dims) - 1) / 2) * h
        g = g[((p / np.array(ELLIPSOID)) ** 2).sum(1) <= 1.0]
        newmark, dt, s0 = True, 5e-5 * (1e6 / n) ** (1 / 3), 0.015
    count = g.shape[0]
    pos, vel, act = np.zeros((count, 4)), np.zeros((count, 4)), np.zeros(count, np.int32)
    pos[:, :3] = (g + rng.uniform(-jitter, jitter, (count, 3))) * h
    stiff = 1e6 * (h / 0.02) ** 2
    if shape == "block":
        act[g[:, 2] == 0] = pd.CLAMPED
        act[g[:, 2] == g[:, 2].max()] = pd.PRESCRIBED
        vel[g[:, 2] == g[:, 2].max(), 2] = -1.0
    elif shape == "beam":
        act[(p[:, 2] < 2 * h) & ((p[:, 0] < 0.05) | (p[:, 0] > 0.95))] = pd.CLAMPED
        load = (p[:, 2] > 0.2 - 2 * h) & (np.abs(p[:, 0] - 0.5) < 0.02)
        act[load] = pd.PRESCRIBED
        vel[load, 2] = -1.0
    else:
        r = 0.5 * R * h if shape == "ball" else RIGID_RADIUS
        mid = 0.0 if shape == "ball" else (np.array(dims) - 1) / 2 * h
        centre = np.zeros(3) + mid
        centre[0] = pos[:, 0].max() + r        # in contact from the first step
        body["sphere"] = (r, centre, (-(5.0 if shape == "ball" else RIGID_SPEED), 0.0, 0.0), stiff / h)
    body.update(sites=g, pos=pos, vel=vel, act=act, h=h, stiff=stiff, mass=1e-3 * (h / 0.02) ** 3, dt=dt, s0=s0,
                newmark=newmark, horizon=coeff * h / 2, n=count)
    return body


def _parameters(b, fp64, guess=0, tolerance=1e-6):
    sp = pd.SystemParameter()
    sim, run, opt = sp.getSimulationParameters(), sp.getRunningParameters(), pd.default_options()
    sim.num_pd_particle = b["n"]
    sim.pd_particle_radius = b["h"] / 2
    sim.pd_kernel_coeff = b["coeff"]
    sim.pd_horizon = b["horizon"]
    sim.pd_particle_mass = b["mass"]
    sim.pd_time_step = 128
    sim.scaleFactor = 1.0
    sim.boundary_min_x = sim.boundary_min_y = sim.boundary_min_z = -1e30
    sim.boundary_max_x = sim.boundary_max_y = sim.boundary_max_z = 1e30
    run.integrator = pd.NEWMARK_BETA if b["newmark"] else pd.IMPLICIT_EULER
    run.adaptive_integration = 0
    run.pd_stretch_limit_s0 = b["s0"]
    run.final_step = 1000
    opt.precision = pd.PRECISION_FP64 if fp64 else pd.PRECISION_MIXED
    opt.cg_relative_tolerance = tolerance
    opt.cg_max_iterations = 20000
    opt.time_step_base = b["dt"] / 128.0
    opt.bond_stiffness = b["stiff"]
    opt.gravity[:] = (0.0, 0.0, -9.81)
    opt.box_enabled = 0
    opt.warm_start = guess
    if b["sphere"]:
        opt.sphere_enabled = 1
        opt.sphere_radius = b["sphere"][0]
        opt.sphere_center[:] = tuple(b["sphere"][1])
        opt.sphere_velocity[:] = b["sphere"][2]
        opt.sphere_stiffness = b["sphere"][3]
    return sim, run, opt


def _simulator(b, fp64, guess=0, tolerance=1e-6):
    s = pd.Simulator(0, *_parameters(b, fp64, guess, tolerance))
    s.get_pd_position()[:] = b["pos"]
    s.get_pd_velocity()[:] = b["vel"]
    s.get_pd_activity()[:] = b["act"]
    return s


def _vector(b, seed):
    x = np.zeros((b["n"], 4))
    x[:, :3] = np.random.default_rng(seed + 1).standard_normal((b["n"], 3)).astype(np.float32)
    return x


# ---- prepare / run ------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "operator":
        b = _body(case["shape"], case["n"], case["coeff"], case["jitter"], seed)
        s = _simulator(b, case["fp64"])
        s.makeReady()
        s.advance(1)   # the operator of a step, at the positions that the step began with
        perm = torch.from_numpy(s.get(pd.VAR_SLOT_PERMUTATION).astype(np.int64)).cuda()
        kind = torch.float64 if case["fp64"] else torch.float32
        x = torch.from_numpy(_vector(b, seed)).to("cuda", kind)[perm].contiguous()
        torch.cuda.synchronize()
        return {"case": case, "sim": s, "x": x, "u": torch.empty_like(x), "v": torch.empty_like(x),
                "slot": torch.argsort(perm), "dot": torch.zeros(1, dtype=torch.float64, device="cuda"),
                "stream": torch.cuda.ExternalStream(s.stream_handle())}
    if case["kind"] == "run":
        b = _body(case["shape"], case["n"], case["coeff"], case["jitter"], seed)
        s = _simulator(b, case["fp64"], case["guess"], case["tolerance"])
        return {"case": case, "sim": s, "position": torch.empty((b["n"], 4), dtype=torch.float64, pin_memory=True),
                "velocity": torch.empty((b["n"], 4), dtype=torch.float64, pin_memory=True)}
    if case["kind"] == "batch":
        batch = pd.Batch(0)
        for k in range(case["count"]):         # sizes spread over their logarithm, large and small in turn
            at = (k * 7 % case["count"]) / max(1, case["count"] - 1)
            n = int(round(case["n"] * (case["n_most"] / case["n"]) ** at))
            b = _body("ball" if k % 2 else "block", n, (4.0, 5.0, 6.0)[k % 3], 0.05, seed * 1000 + k)
            batch.add_scene(*_parameters(b, False, 0, case["tolerance"]), b["pos"], b["vel"], b["act"])
        return {"case": case, "batch": batch}
    X, T, params = _network(case, seed)
    return {"case": case, "X": X, "T": T, "params": params}


def run(state):
    case = state["case"]
    if case["kind"] == "operator":
        s, x, y, z = state["sim"], state["x"], state["u"], state["v"]
        for _ in range(PRODUCTS):
            s.apply_operator(x.data_ptr(), y.data_ptr(), state["dot"].data_ptr())
            x, y, z = y, z, y
        with torch.cuda.stream(state["stream"]):   # the caller's particle order, whole rows of 16 (32) bytes at a time
            rows = x.view(torch.complex128).reshape(x.shape[0], -1)
            rows = rows.reshape(-1)[state["slot"]] if rows.shape[1] == 1 else rows.index_select(0, state["slot"])
            return {"y": torch.view_as_real(rows).view(x.dtype).reshape(x.shape), "dot": state["dot"].to(x.dtype)}
    if case["kind"] == "run":
        s, x, v = state["sim"], state["position"], state["velocity"]
        s.makeReady()
        for done in range(0, case["steps"], case["frame"]):
            s.advance(min(case["frame"], case["steps"] - done))
            s.get(pd.VAR_POSITION, out=x.numpy())
        out = {"position": x if case["fp64"] else x.float(), "bonds": s.get(pd.VAR_BOND_COUNT)}
        # (Newmark's velocities, 2 dx / h - v, carry the rounding of 32-bit
        # solutions undamped from step to step: a program takes the positions)
        if case["fp64"] or case["shape"] == "block":
            s.get(pd.VAR_VELOCITY, out=v.numpy())
            out["velocity"] = v if case["fp64"] else v.float()
        return out
    if case["kind"] == "batch":
        b = state["batch"]
        b.makeReady()
        b.advance(case["steps"])
        return {what: np.concatenate([b.get(k, var) for k in range(case["count"])]).astype(kind)
                for what, var, kind in (("position", pd.VAR_POSITION, np.float32), ("bonds", pd.VAR_BOND_COUNT, np.int32))}
    if case["grad"]:
        loss, grad = pd.mlp_loss_grad(state["X"], state["T"], state["params"])
        return {"loss": np.float32(loss), "grad": grad}
    return {"y": pd.mlp_predict(state["X"], state["params"])}


# ---- what a pass cannot do without --------------------------------------------------
BONDS = {4.0: 29, 5.0: 76, 6.0: 104}           # live bonds per particle, about
SOLVES = {"block": 50, "ball": 70, "beam": 225, "ellipsoid": 350}   # CG iterations per step, about


def _product(n, bonds, fp64):
    """One product A x: a neighbour index or rest length per bond, positions, x and y per particle."""
    return {"bytes": n * ((4 * bonds + 128) if fp64 else (4 * bonds + 64)), "flops": 30 * n * bonds}


def work(case):
    if case["kind"] == "operator":
        return {k: PRODUCTS * v for k, v in _product(case["n"], BONDS[case["coeff"]], case["fp64"]).items()}
    if case["kind"] == "network":
        rows, macs = case["rows"], 64 * 128 + 128 * 128 + 128 * 3
        return {"bytes": rows * (64 + 3) * 4, "flops": rows * macs * (6 if case["grad"] else 2)}
    if case["kind"] == "batch":
        n = case["count"] * 0.5 * (case["n"] + case["n_most"])
        bonds, solves, fp64 = 70, 60, False
    else:
        n, bonds, fp64 = case["n"], BONDS[case["coeff"]], case["fp64"]
        solves = SOLVES[case["shape"]] * (2 if fp64 else 1)
    one, vectors = _product(n, bonds, fp64), n * (288 if fp64 else 144)
    return {"bytes": case["steps"] * solves * (one["bytes"] + vectors), "flops": case["steps"] * solves * one["flops"]}


# ---- 64-bit values ------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "operator":
        return _exact_operator(case, seed)
    if case["kind"] == "network":
        return _exact_network(case, seed)
    return None     # hundreds of solves


def _exact_operator(case, seed):
    """m w_p + beta h^2 [c sum_q (xi . (w_p - w_q)) xi / d^3 + k (n . w_p) n] over
    the bonds of the undeformed body and its particles in contact, four times."""
    b = _body(case["shape"], case["n"], case["coeff"], case["jitter"], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.from_numpy(b["pos"][:, :3].copy()).to(dev)
    w = torch.from_numpy(_vector(b, seed)[:, :3].copy()).to(dev)
    free = torch.from_numpy(b["act"] == pd.ACTIVE).to(dev)[:, None]    # the other rows are Dirichlet rows
    reach = int(math.floor(case["coeff"] / 2 + 2 * case["jitter"]))
    g = torch.from_numpy(b["sites"]).to(dev)
    g = g - g.min(0).values + reach
    dim = (g.max(0).values + reach + 1).tolist()
    at = torch.full((dim[0] * dim[1] * dim[2],), -1, dtype=torch.int64, device=dev)
    here = (g[:, 2] * dim[1] + g[:, 1]) * dim[0] + g[:, 0]
    at[here] = torch.arange(b["n"], device=dev)
    t2 = b["dt"] ** 2 / (4.0 if b["newmark"] else 1.0)
    touch, normal = torch.zeros((b["n"], 1), dtype=torch.bool, device=dev), X
    if b["sphere"]:
        radius, centre, _, stiff = b["sphere"]
        normal = X - torch.from_numpy(centre).to(dev)
        far = normal.norm(dim=1, keepdim=True)
        touch, normal = far < radius + b["h"] / 2, normal / far
    steps = range(-reach, reach + 1)
    for _ in range(PRODUCTS):
        acc = torch.zeros_like(w)
        for dz in steps:
            for dy in steps:
                for dx in steps:
                    if dx == dy == dz == 0:
                        continue
                    q = at[here + (dz * dim[1] + dy) * dim[0] + dx]
                    p = torch.nonzero(q >= 0).reshape(-1)
                    q = q[p]
                    xi = X[q] - X[p]
                    d = (xi * xi).sum(1).sqrt()
                    on = d < b["horizon"]
                    p, q, xi, d = p[on], q[on], xi[on], d[on]
                    acc.index_add_(0, p, ((xi * (w[p] - w[q])).sum(1) / d ** 3)[:, None] * xi)
        acc *= b["stiff"]
        if b["sphere"]:
            acc += torch.where(touch, stiff * (normal * w).sum(1, keepdim=True) * normal, 0.0)
        y = torch.where(free, b["mass"] * w + t2 * acc, 0.0)
        dot = (y * w).sum().reshape(1)
        w = y
    return {"y": torch.cat([y, torch.zeros_like(y[:, :1])], 1), "dot": dot}


def _network(case, seed):
    """Normalised features, targets and Glorot-uniform parameters."""
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((case["rows"], 64)).astype(np.float32)
    T = rng.standard_normal((case["rows"], 3)).astype(np.float32)
    parts = []
    for a, b in ((64, 128), (128, 128), (128, 3)):
        lim = math.sqrt(6 / (a + b))
        parts += [rng.uniform(-lim, lim, a * b), rng.uniform(-0.1, 0.1, b)]
    return X, T, np.concatenate(parts).astype(np.float32)


def _exact_network(case, seed):
    X, T, params = (torch.from_numpy(v).double() for v in _network(case, seed))
    params.requires_grad_(case["grad"])
    h, i = X, 0
    for k, (a, b) in enumerate(((64, 128), (128, 128), (128, 3))):
        z = h @ params[i:i + a * b].reshape(a, b) + params[i + a * b:i + a * b + b]
        h = z if k == 2 else 0.5 * z * (1 + torch.erf(z / math.sqrt(2)))
        i += a * b + b
    if not case["grad"]:
        return {"y": h}
    loss = ((h - T) ** 2).sum(1).mean()
    loss.backward()
    return {"loss": loss.detach(), "grad": params.grad}
