"""Performance cases of the particle-mesh framework: what its users run, through its public entry points.

Each case is a dict of plain values; ``prepare`` builds what a program holds before the call, ``run`` is
one call, ``work`` the bytes and operations the call cannot do without, ``exact`` the same outputs from
plain torch in 64 bits. The kinds:

* ``advance``  -- one KDK step of a running simulation (``PMEngine.advance`` / ``advance_graph``);
* ``simulate`` -- a whole short run from host arrays to host arrays (load, steps, export);
* ``kdk``      -- one step of the reference-shaped chain: ``kdk_step`` over deposit, multigrid solve,
  gradient and gather, on particles in the caller's order;
* ``solve``    -- a cold multigrid solve of a density (``MultigridPoissonSolver.solve``);
* ``forward``, ``train`` -- the warm-start network: inference, and one training step;
* ``diagnostics`` -- one conservation sample (``DeviceDiagnostics.sample``).
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PACKAGE = ROOT / "galaxy-collision-with-cuda-fft_gb300"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

BOX = 64.0      # two-disk box edge
WARM_STEPS = 3  # steps taken before a measured one: the warm-start history is complete


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # The Plummer configuration (configs/plummer_131k.yaml): the smallest simulation, driven step by
        # step as run_simulation does, each solve started from the previous potential.
        {"name": "plummer_131k", "kind": "advance", "model": "plummer", "n": 131072, "grid": 64, "box": 24.0,
         "dt": 0.01, "bits": 52, "guess": "plain", "graph": False, "phases": False},
        # One large member of the collision ensemble: 128^3, learned initial guess, replayed step graph.
        {"name": "member_2M", "kind": "advance", "model": "two_disk", "n": 1873211, "grid": 128, "box": BOX,
         "dt": 0.005, "bits": 40, "guess": "learned", "graph": True, "phases": True},
        # configs/two_disk_10M.yaml: as much grid as particle work.
        {"name": "two_disk_10M", "kind": "advance", "model": "two_disk", "n": 10000000, "grid": 256, "box": BOX,
         "dt": 0.005, "bits": 44, "guess": "extrapolate", "graph": True, "phases": False},
        # configs/two_disk_100M.yaml: the headline workload.
        {"name": "two_disk_100M", "kind": "advance", "model": "two_disk", "n": 100000000, "grid": 256, "box": BOX,
         "dt": 0.005, "bits": 40, "guess": "extrapolate", "graph": True, "phases": False},
        # A short run end to end with an odd particle count, a grid that is no power of two and a spacing
        # that is not exact in binary: pinned host arrays in, pinned host arrays out.
        {"name": "run_1M5_100", "kind": "simulate", "n": 1500001, "grid": 100, "dt": 0.005, "steps": 20,
         "bits": 52, "guess": "extrapolate"},
        # The drop-in chain of a program written against the reference, small ...
        {"name": "kdk_250k_64", "kind": "kdk", "model": "two_disk", "n": 250000, "grid": 64, "box": BOX,
         "dt": 0.005, "tol": 1e-6},
        # ... and at the 10M configuration.
        {"name": "kdk_10M_256", "kind": "kdk", "model": "two_disk", "n": 10000000, "grid": 256, "box": BOX,
         "dt": 0.005, "tol": 1e-6},
        # A potential from scratch (initial conditions, analysis of snapshots), at the production grid ...
        {"name": "solve_256", "kind": "solve", "grid": 256, "tol": 1e-6},
        # ... and on an odd grid.
        {"name": "solve_97", "kind": "solve", "grid": 97, "tol": 1e-6},
        # The network behind the learned guess at a 256^3 grid, and a training step at half that size.
        {"name": "forward_128", "kind": "forward", "R": 128},
        {"name": "train_64", "kind": "train", "R": 64},
        # A conservation sample of the 10M run (taken at every output step).
        {"name": "diagnostics_10M", "kind": "diagnostics", "n": 10000000, "grid": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("advance", "advance", "advance", "simulate", "kdk", "kdk", "solve", "solve", "forward", "train",
                       "diagnostics"))
    dt = round(rng.uniform(0.002, 0.008), 5)
    if kind == "advance":
        guess = rng.choice(("plain", "extrapolate", "extrapolate", "learned"))
        grid = 16 * rng.randint(4, 16) if guess == "learned" else rng.choice((64, 80, 96, 100, 128, 150, 192, 256))
        return {"kind": kind, "model": "two_disk", "n": _log_int(rng, 1e5, 6e7), "grid": grid, "box": BOX, "dt": dt,
                "bits": rng.choice((40, 44, 52)), "guess": guess, "graph": rng.random() < 0.7,
                "phases": rng.random() < 0.3}
    if kind == "simulate":
        return {"kind": kind, "n": _log_int(rng, 1e5, 4e6), "grid": rng.choice((64, 90, 100, 128, 200)), "dt": dt,
                "steps": rng.randint(5, 25), "bits": 52, "guess": rng.choice(("plain", "extrapolate"))}
    if kind == "kdk":
        model = rng.choice(("plummer", "two_disk"))
        return {"kind": kind, "model": model, "n": _log_int(rng, 5e4, 2e7),
                "grid": rng.choice((50, 64, 97, 128, 192, 256)), "box": 24.0 if model == "plummer" else BOX, "dt": dt,
                "tol": rng.choice((1e-3, 1e-6))}
    if kind == "solve":
        return {"kind": kind, "grid": _log_int(rng, 40, 256), "tol": rng.choice((1e-3, 1e-6, 1e-8))}
    if kind == "forward":
        return {"kind": kind, "R": 8 * rng.randint(4, 16)}
    if kind == "train":
        return {"kind": kind, "R": 8 * rng.randint(4, 12)}
    return {"kind": kind, "n": _log_int(rng, 1e5, 2e7), "grid": rng.choice((64, 128, 256))}


# ------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(shape, device="cuda", generator=g)


def _randn(g, *shape):
    return torch.randn(shape, device="cuda", generator=g)


def _disk(g, n, mass, rd, soft, incline):
    """n - 1 particles of a truncated exponential sech^2 disk and its central point mass (the last one)."""
    nd = n - 1
    table = torch.linspace(0.0, 5.0 * rd, 4097, device="cuda", dtype=torch.float64)
    cdf = 1.0 - (1.0 + table / rd) * torch.exp(-table / rd)
    cdf = (cdf / cdf[-1].clone()).float()
    table = table.float()
    u = _rand(g, nd)
    j = torch.clamp(torch.searchsorted(cdf, u) - 1, 0, 4095)
    r = table[j] + (u - cdf[j]) / (cdf[j + 1] - cdf[j]) * (table[j + 1] - table[j])
    del j
    theta = _rand(g, nd) * (2.0 * math.pi)
    z = 0.1 * rd * torch.atanh(torch.clamp(2.0 * _rand(g, nd) - 1.0, -0.999999, 0.999999))
    m_bh = 0.01 * mass
    vc = torch.sqrt((mass * u + m_bh) * r * r / (r * r + soft * soft) ** 1.5)
    del u
    c, s = torch.cos(theta), torch.sin(theta)
    del theta
    pos = torch.zeros((n, 3), device="cuda")
    vel = torch.zeros((n, 3), device="cuda")
    pos[:nd, 0], pos[:nd, 1], pos[:nd, 2] = r * c, r * s, z
    for a, rot in enumerate((-vc * s, vc * c, None)):
        vel[:nd, a] = 0.1 * vc * _randn(g, nd)
        if rot is not None:
            vel[:nd, a] += rot
    if incline:
        t = math.radians(incline)
        ct, st = math.cos(t), math.sin(t)
        for w in (pos, vel):
            y, zz = w[:, 1].clone(), w[:, 2].clone()
            w[:, 1], w[:, 2] = ct * y - st * zz, st * y + ct * zz
    m = torch.full((n,), mass / nd, device="cuda")
    m[-1] = m_bh
    return pos, vel, m


def _two_disk(n, dx, seed):
    g = _gen(seed)
    n1 = max(2, int(0.4 * n))
    sep, approach = (20.0, 2.0, 0.0), 0.5
    parts = [_disk(g, n1, 1.0, 1.0, dx, 0.0), _disk(g, n - n1, 1.5, 1.2, dx, 30.0)]
    for (pos, vel, _), w in zip(parts, (-0.6, 0.4)):
        pos += torch.tensor([w * s for s in sep], device="cuda")
        vel[:, 0] -= w * approach
    gid = torch.zeros(n, dtype=torch.int32, device="cuda")
    gid[n1:] = 1
    return [torch.cat([p[k] for p in parts]) for k in range(3)] + [gid]


def _plummer(n, seed):
    g = _gen(seed)

    def directions():
        v = _randn(g, n, 3)
        return v / v.norm(dim=1, keepdim=True)

    u = _rand(g, n).double() * 0.985 + 1e-9  # r <= 10
    r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    q = torch.linspace(0.0, 1.0, 8193, device="cuda", dtype=torch.float64)
    w = torch.cumsum(q**2 * (1.0 - q**2) ** 3.5, 0)
    speed = q[torch.clamp(torch.searchsorted(w / w[-1], _rand(g, n).double()), 0, 8192)]
    speed = speed * math.sqrt(2.0) * (1.0 + r * r) ** (-0.25)
    pos = (r[:, None] * directions().double()).float()
    vel = (speed[:, None] * directions().double()).float()
    return [pos, vel, torch.full((n,), 1.0 / n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")]


def _particles(case, seed):
    """pos (n, 3), vel (n, 3) in physical coordinates, mass, gid."""
    dx = case.get("box", BOX) / case["grid"]
    return _plummer(case["n"], seed) if case.get("model") == "plummer" else _two_disk(case["n"], dx, seed)


def _spacing(case):
    box = case.get("box", BOX)
    return box / case["grid"], -box / 2.0


def _density(case, seed):
    """The density of a two-disk system of about two particles per node of the smaller grids (f32)."""
    dx, lo = _spacing(case)
    pos, _, m, _ = _two_disk(min(4_000_000, 2 * case["grid"] ** 3), dx, seed)
    x = pos.double() - lo
    return _deposit64([x[:, a] for a in range(3)], m.double(), case["grid"], dx).float()


def _network_inputs(case, seed):
    """Smooth random fields of unit scale, as the network's inputs and target are (f16)."""
    g, R = _gen(seed), case["R"]

    def field(scale):
        low = _randn(g, 1, 1, 8, 8, 8)
        f = torch.nn.functional.interpolate(low, size=(R, R, R), mode="trilinear", align_corners=True)[0, 0]
        return scale * (f + 0.1 * _randn(g, R, R, R))

    feat = torch.stack([torch.log1p(field(1.0).abs() * 4.0), field(1.0) - 0.8, field(1.0), field(1.0)])
    return feat.half().contiguous(), field(0.7).half().contiguous()


# ------------------------------------------------------------------------------ preparation
def prepare(case, seed):
    return {"advance": _prepare_advance, "simulate": _prepare_simulate, "kdk": _prepare_kdk, "solve": _prepare_solve,
            "forward": _prepare_network, "train": _prepare_network, "diagnostics": _prepare_diagnostics}[case["kind"]](
                case, seed)


def _engine(case):
    from galaxy_collision_gb300.engine import PMEngine
    from galaxy_collision_gb300.warmstart import WarmStartNet

    dx, lo = _spacing(case)
    eng = PMEngine(case["grid"], dx, origin=(lo,) * 3, tol=1e-6, fixed_point_bits=case["bits"],
                   phase_launches=case.get("phases", False))
    eng.set_warmstart(case["guess"],
                      net=WarmStartNet.load(R=case["grid"] // 2) if case["guess"] == "learned" else None)
    return eng


def _prepare_advance(case, seed):
    pos, vel, m, gid = _particles(case, seed)
    eng = _engine(case)
    eng.load(pos, vel, m, gid)
    eng.prime(case["dt"])
    for _ in range(WARM_STEPS):
        eng.advance(case["dt"])
    if case["graph"]:
        eng.prepare_graphs(case["dt"])
    return {"case": case, "eng": eng}


def _prepare_simulate(case, seed):
    pos, vel, m, gid = _particles(case, seed)
    host = [t.cpu().pin_memory() for t in (pos, vel, m, gid)]
    eng = _engine(case)
    eng.reserve(case["n"])
    out = [torch.empty((case["n"], 3), dtype=torch.float32, pin_memory=True) for _ in range(2)]
    return {"case": case, "eng": eng, "host": host, "out": out}


def _particle_state(pos, vel, m, gid, lo):
    from galaxy_collision_gb300.data import ParticleState

    parts = ParticleState(int(m.numel()))
    x = (pos.double() - lo).float()
    for a, k in enumerate("xyz"):
        getattr(parts, "pos_" + k).tensor.copy_(x[:, a])
        getattr(parts, "vel_" + k).tensor.copy_(vel[:, a])
    parts.mass.tensor.copy_(m)
    parts.gid.tensor.copy_(gid)
    return parts


def _prepare_kdk(case, seed):
    from galaxy_collision_gb300.data import Field, GridState
    from galaxy_collision_gb300.deposit import deposit_density, gather_acceleration, potential_to_accel
    from galaxy_collision_gb300.solver import make_solver

    dx, lo = _spacing(case)
    parts = _particle_state(*_particles(case, seed), lo)
    grid = GridState(case["grid"])
    acc = [Field(case["n"]) for _ in range(3)]
    solver = make_solver("multigrid", case["grid"], dx=dx, grav_constant=1.0, tol=case["tol"])
    first = [True]

    def accel():
        deposit_density(parts, grid.rho, dx)
        solver.solve(grid.rho, grid.phi, warm_start=not first[0])
        first[0] = False
        potential_to_accel(grid.phi, grid.ax, grid.ay, grid.az, dx)
        gather_acceleration(parts, grid.ax, grid.ay, grid.az, *acc, dx)

    accel()
    return {"case": case, "parts": parts, "grid": grid, "acc": acc, "accel": accel}


def _prepare_solve(case, seed):
    from galaxy_collision_gb300.solver import make_solver

    rho = _density(case, seed)
    return {"case": case, "rho": rho, "phi": torch.zeros_like(rho),
            "solver": make_solver("multigrid", case["grid"], dx=_spacing(case)[0], grav_constant=1.0,
                                  tol=case["tol"])}


def _prepare_network(case, seed):
    from galaxy_collision_gb300.warmstart import WarmStartNet

    feat, target = _network_inputs(case, seed)
    return {"case": case, "net": WarmStartNet.load(R=case["R"]), "feat": feat, "target": target}


def _diagnostics_inputs(case, seed):
    dx, lo = _spacing(case)
    pos, vel, m, gid = _two_disk(case["n"], dx, seed)
    vel += torch.tensor([0.1, 0.05, -0.02], device="cuda")  # the system drifts: its momentum is not a rounding error
    g = _gen(seed + 7)
    G = case["grid"]
    rho = torch.exp(_randn(g, G, G, G))
    phi = -1.0 - _rand(g, G, G, G)
    return (pos, vel, m, gid), lo, rho, phi


def _prepare_diagnostics(case, seed):
    from galaxy_collision_gb300.data import GridState
    from galaxy_collision_gb300.diagnostics_device import DeviceDiagnostics

    ic, lo, rho, phi = _diagnostics_inputs(case, seed)
    grid = GridState(case["grid"])
    grid.rho.tensor.copy_(rho)
    grid.phi.tensor.copy_(phi)
    diag = DeviceDiagnostics(case["grid"], r_max=BOX * math.sqrt(3.0))
    return {"case": case, "parts": _particle_state(*ic, lo), "grid": grid, "diag": diag}


# ------------------------------------------------------------------------------ one pass
def run(state):
    return {"advance": _run_advance, "simulate": _run_simulate, "kdk": _run_kdk, "solve": _run_solve,
            "forward": _run_forward, "train": _run_train, "diagnostics": _run_diagnostics}[state["case"]["kind"]](state)


def _run_advance(s):
    eng, case = s["eng"], s["case"]
    if case["graph"]:
        eng.advance_graph(case["dt"])
    else:
        eng.advance(case["dt"])
    return {k: eng.cur[k] for k in ("x", "y", "z", "vx", "vy", "vz", "pid")}


def _run_simulate(s):
    eng, case = s["eng"], s["case"]
    eng.load(*s["host"])
    eng.run(case["steps"], case["dt"])
    pos, vel, _, _ = eng.export(*s["out"])
    return {"pos": pos, "vel": vel}


def _run_kdk(s):
    from galaxy_collision_gb300.integrator import kdk_step

    p, g = s["parts"], s["grid"]
    kdk_step(p, *s["acc"], s["accel"], s["case"]["dt"])
    out = {k: getattr(p, k).tensor for k in ("pos_x", "pos_y", "pos_z", "vel_x", "vel_y", "vel_z")}
    out.update(zip(("acc_x", "acc_y", "acc_z"), (a.tensor for a in s["acc"])))
    out["rho"], out["phi"] = g.rho.tensor, g.phi.tensor
    return out


def _run_solve(s):
    s["solver"].solve(s["rho"], s["phi"], warm_start=False)
    return {"phi": s["phi"]}


def _run_forward(s):
    return {"y": s["net"].forward(s["feat"])}


def _run_train(s):
    net = s["net"]
    y = net.forward(s["feat"])
    loss = net.backward(s["target"])
    grads = net.grads()
    net.adam_step(1e-3)
    return {"y": y, "loss": loss, "grads": grads, "params": net.params()}


def _run_diagnostics(s):
    return s["diag"].sample(s["parts"], s["grid"], _spacing(s["case"])[0])


# ------------------------------------------------------------------------------ what a pass cannot do without
def _layers():
    """(cin, cout, level) of the network's convolutions."""
    return ((16, 16, 0), (16, 32, 1), (32, 64, 2), (64, 128, 3), (128, 64, 3), (64, 64, 2), (64, 32, 2), (32, 32, 1),
            (32, 16, 1), (16, 16, 0), (16, 16, 0))


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        flops = sum(54.0 * ci * co * (case["R"] >> lv) ** 3 for ci, co, lv in _layers())
        params = sum(27 * ci * co + co for ci, co, _ in _layers())
        if kind == "forward":
            return {"bytes": 12.0 * case["R"] ** 3 + 4.0 * params, "flops": flops}
        return {"bytes": 14.0 * case["R"] ** 3 + 28.0 * params, "flops": 3.0 * flops}
    G3 = float(case["grid"]) ** 3
    if kind == "solve":  # density in, potential out; a handful of operations a node and cycle
        return {"bytes": 8.0 * G3, "flops": 40.0 * G3 * -math.log10(case["tol"])}
    n = float(case["n"])
    if kind == "diagnostics":
        return {"bytes": 28.0 * n + 8.0 * G3, "flops": 60.0 * n + 2.0 * G3}
    if kind == "kdk":  # state in and out, accelerations in and out; rho, phi and the acceleration grids out, phi in
        return {"bytes": 76.0 * n + 24.0 * G3, "flops": 200.0 * n + 40.0 * G3 * -math.log10(case["tol"])}
    step = {"bytes": 52.0 * n + 16.0 * G3, "flops": 200.0 * n + 240.0 * G3}  # x, v, m in, x, v out; potential in, out
    if kind == "simulate":
        return {"bytes": case["steps"] * step["bytes"] + 56.0 * n, "flops": case["steps"] * step["flops"]}
    return step


# ------------------------------------------------------------------------------ the same outputs in 64 bits
CHUNK = 1 << 22


def _cells(x, dx, n):
    """Lower cell index and weights along each axis for particles inside the grid."""
    g = [c / dx for c in x]
    i = [torch.floor(c) for c in g]
    f = [c - b for c, b in zip(g, i)]
    return [b.long() for b in i], f


def _corners(x, dx, n):
    """(node index, weight) of the eight corners; corners outside the grid have weight 0."""
    i, f = _cells(x, dx, n)
    for c in range(8):
        o = (c >> 2, (c >> 1) & 1, c & 1)
        node, w, inside = 0, 1.0, True
        for a in range(3):
            j = i[a] + o[a]
            inside = inside & (j >= 0) & (j < n)
            node = node * n + torch.clamp(j, 0, n - 1)
            w = w * (f[a] if o[a] else 1.0 - f[a])
        yield node, torch.where(inside, w, torch.zeros_like(w))


def _deposit64(x, m, n, dx):
    rho = torch.zeros(n**3, dtype=torch.float64, device="cuda")
    for s in range(0, m.numel(), CHUNK):
        for node, w in _corners([c[s:s + CHUNK] for c in x], dx, n):
            rho.index_add_(0, node, w * m[s:s + CHUNK])
    return rho.view(n, n, n) / dx**3


def _faces64(rho, dx):
    """Monopole + quadrupole potential of rho about its centre of mass, at every node (G = 1)."""
    n = rho.shape[0]
    t = torch.arange(n, dtype=torch.float64, device="cuda") * dx
    m = rho * dx**3
    M = m.sum()
    s = [m.sum((1, 2)), m.sum((0, 2)), m.sum((0, 1))]
    c = [(q * t).sum() / M for q in s]
    d = [t - q for q in c]
    S = [[None] * 3 for _ in range(3)]
    for a in range(3):
        S[a][a] = (s[a] * d[a] ** 2).sum()
        for b in range(a + 1, 3):
            S[a][b] = (m.sum(3 - a - b) * d[a][:, None] * d[b][None, :]).sum()
    r = (d[0][:, None, None], d[1][None, :, None], d[2][None, None, :])
    d2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2 + 1e-12
    q = sum(S[a][a] * r[a] ** 2 for a in range(3))
    q = q + 2.0 * sum(S[a][b] * r[a] * r[b] for a in range(3) for b in range(a + 1, 3))
    quad = 3.0 * q / d2 - (S[0][0] + S[1][1] + S[2][2])
    return -(M / torch.sqrt(d2) + 0.5 * quad / d2**1.5)


def _solve64(rho, dx):
    """The exact solution of the 7-point problem laplacian(phi) = 4 pi rho with those faces (sine transforms)."""
    n = rho.shape[0]
    phi = _faces64(rho, dx)
    phi[1:-1, 1:-1, 1:-1] = 0.0
    b = 4.0 * math.pi * dx * dx * rho[1:-1, 1:-1, 1:-1]
    b = b.clone()
    b[0] -= phi[0, 1:-1, 1:-1]
    b[-1] -= phi[-1, 1:-1, 1:-1]
    b[:, 0] -= phi[1:-1, 0, 1:-1]
    b[:, -1] -= phi[1:-1, -1, 1:-1]
    b[:, :, 0] -= phi[1:-1, 1:-1, 0]
    b[:, :, -1] -= phi[1:-1, 1:-1, -1]
    k = torch.arange(1, n - 1, dtype=torch.float64, device="cuda")
    S = torch.sin(torch.outer(k, k) * (math.pi / (n - 1)))
    lam = 2.0 * torch.cos(k * (math.pi / (n - 1))) - 2.0

    def transform(v):
        for _ in range(3):
            v = torch.tensordot(v, S, dims=([0], [0]))  # the transformed axis moves last: three turns restore the order
        return v

    b = transform(b) / (lam[:, None, None] + lam[None, :, None] + lam[None, None, :])
    phi[1:-1, 1:-1, 1:-1] = transform(b) * (2.0 / (n - 1)) ** 3
    return phi


def _minus_grad64(phi, dx):
    out = []
    for a in range(3):
        p = phi.movedim(a, 0)
        g = torch.empty_like(p)
        g[1:-1] = (p[2:] - p[:-2]) / (2.0 * dx)
        g[0], g[-1] = (p[1] - p[0]) / dx, (p[-1] - p[-2]) / dx
        out.append(-g.movedim(0, a).contiguous())
    return out


def _gather64(x, field, dx):
    n = field[0].shape[0]
    out = [torch.zeros_like(x[0]) for _ in range(3)]
    flat = [f.reshape(-1) for f in field]
    for s in range(0, x[0].numel(), CHUNK):
        for node, w in _corners([c[s:s + CHUNK] for c in x], dx, n):
            for o, f in zip(out, flat):
                o[s:s + CHUNK] += w * f[node]
    return out


def _force64(x, m, n, dx):
    rho = _deposit64(x, m, n, dx)
    phi = _solve64(rho, dx)
    return rho, phi, _gather64(x, _minus_grad64(phi, dx), dx)


def _start64(case, seed):
    """Positions (from the grid origin, as rounded to f32), velocities and masses in 64 bits."""
    pos, vel, m, _ = _particles(case, seed)
    lo = _spacing(case)[1]
    x = (pos.double() - lo).float()
    return ([x[:, a].double().contiguous() for a in range(3)], [vel[:, a].double().contiguous() for a in range(3)],
            m.double(), x)


def _kick64(v, a, t):
    for q, b in zip(v, a):
        q += b * t


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        return _exact_network(case, seed)
    if kind == "diagnostics":
        return _exact_diagnostics(case, seed)
    dx, lo = _spacing(case)
    if kind == "solve":
        return {"phi": _solve64(_density(case, seed).double(), dx)}
    n, dt = case["grid"], case["dt"]
    evaluations = {"advance": WARM_STEPS + 2, "kdk": 2}.get(kind) or case["steps"] + 1
    if case["n"] * evaluations > 100_000_000:
        return None
    x, v, m, x32 = _start64(case, seed)
    rho, phi, a = _force64(x, m, n, dx)
    if kind == "kdk":
        _kick64(v, a, 0.5 * dt)
        _kick64(x, v, dt)
        rho, phi, a = _force64(x, m, n, dx)
        _kick64(v, a, 0.5 * dt)
        out = dict(zip(("pos_x", "pos_y", "pos_z", "vel_x", "vel_y", "vel_z", "acc_x", "acc_y", "acc_z"), x + v + a))
        return out | {"rho": rho, "phi": phi}
    # load, prime, then steps that close the previous one and open their own
    _kick64(v, a, 0.5 * dt)
    _kick64(x, v, dt)
    for _ in range(evaluations - 2):
        _, _, a = _force64(x, m, n, dx)
        _kick64(v, a, dt)
        _kick64(x, v, dt)
    _, _, a = _force64(x, m, n, dx)
    if kind == "simulate":
        _kick64(v, a, 0.5 * dt)
        return {"pos": torch.stack(x, 1) + lo, "vel": torch.stack(v, 1)}
    _kick64(v, a, dt)
    _kick64(x, v, dt)
    # the engine keeps its particles in the order of their cells when loaded
    cell = torch.floor(x32 / torch.tensor(dx, dtype=torch.float32, device="cuda")).long() + 1
    order = torch.sort((cell[:, 0] * (n + 1) + cell[:, 1]) * (n + 1) + cell[:, 2], stable=True).indices
    return dict(zip(("x", "y", "z", "vx", "vy", "vz"), (q[order] for q in x + v))) | {"pid": None}


def _exact_diagnostics(case, seed):
    dx, _ = _spacing(case)
    (pos, vel, m, _), lo, rho, phi = _diagnostics_inputs(case, seed)
    x = (pos.double() - lo).float().double()
    v, m = vel.double(), m.double()
    total = m.sum()
    com = (m[:, None] * x).sum(0) / total
    ke = 0.5 * (m * (v * v).sum(1)).sum()
    pe = 0.5 * dx**3 * (rho.double() * phi.double()).sum()
    # half of the mass, linear within its bin of the same 2048 radial bins
    width = BOX * math.sqrt(3.0) / 2048
    c32 = com.float().double()
    b = torch.clamp((torch.sqrt(((x - c32) ** 2).sum(1)) * float(np.float32(1.0 / width))).long(), 0, 2047)
    hist = torch.zeros(2048, dtype=torch.float64, device="cuda").index_add_(0, b, m).cpu().numpy()
    cum = np.cumsum(hist)
    k = int(np.searchsorted(cum, 0.5 * float(total)))
    below = cum[k - 1] if k else 0.0
    half = (k + (0.5 * float(total) - below) / hist[k]) * width
    return {"M": float(total), "kinetic": float(ke), "potential": float(pe), "energy": float(ke + pe),
            "momentum": (m[:, None] * v).sum(0).cpu().numpy(),
            "ang_momentum": (m[:, None] * torch.linalg.cross(x, v)).sum(0).cpu().numpy(),
            "center_of_mass": com.cpu().numpy(), "half_mass_radius": half}


def _exact_network(case, seed):
    """The network in 64 bits from its stored 32-bit parameters (no bf16 anywhere)."""
    import torch.nn.functional as F

    if case["kind"] == "train" and case["R"] > 80:
        return None
    feat, target = _network_inputs(case, seed)
    with np.load(PACKAGE / "galaxy_collision_gb300" / "warmstart_weights.npz") as z:
        params = torch.from_numpy(z["params"]).cuda().double().requires_grad_(case["kind"] == "train")
    w, at = [], 0
    for ci, co, _ in _layers():
        k = 27 * ci * co
        w.append((params[at:at + k].view(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2), params[at + k:at + k + co]))
        at += k + co

    def conv(l, v):
        return F.conv3d(v, w[l][0], w[l][1], padding=1)

    def up(v):
        return v.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    x0 = F.pad(feat.double()[None], (0, 0, 0, 0, 0, 0, 0, 12))
    e0 = F.relu(conv(0, x0))
    e1 = F.relu(conv(1, F.avg_pool3d(e0, 2)))
    e2 = F.relu(conv(2, F.avg_pool3d(e1, 2)))
    e3 = F.relu(conv(3, F.avg_pool3d(e2, 2)))
    f2 = F.relu(conv(5, F.relu(up(conv(4, e3)) + e2)))
    f1 = F.relu(conv(7, F.relu(up(conv(6, f2)) + e1)))
    f0 = F.relu(conv(9, F.relu(up(conv(8, f1)) + e0)))
    y = conv(10, f0)[0, 0]
    if case["kind"] == "forward":
        return {"y": y}
    loss = 0.5 * ((y - target.double()) ** 2).mean()
    (g,) = torch.autograd.grad(loss, params)
    return {"y": y.detach(), "loss": loss.detach().view(1), "grads": g, "params": None}
