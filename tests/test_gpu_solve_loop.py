"""The eager solve's loop as a graph of the context (from the second solve with the same
parameters on) against the host loop (per-kernel profiling takes it): the same potential,
cycles, verdict and norms."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rho(n, kind):
    g = torch.Generator(device="cuda").manual_seed(n)
    r = torch.rand((n, n, n), device="cuda", generator=g) ** 5
    return torch.zeros_like(r) if kind == "empty" else r


@pytest.mark.parametrize("n", [16, 64, 97, 144])
@pytest.mark.parametrize("kw", [dict(tol=1e-6), dict(tol=1e-3, min_cycles=3), dict(tol=0.0, n_cycles=4),
                                dict(tol=1e-6, n_cycles=1), dict(tol=1e-7, natural_layout=True)])
@pytest.mark.parametrize("kind", ["random", "empty"])
def test_graph_loop_equals_host_loop(cuda, n, kw, kind):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    rho = _rho(n, kind)
    s = MultigridPoissonSolver(n, dx=0.5, grav_constant=1.0, **{"n_cycles": 30, **kw})
    seen = []
    for mode in ("host", "first", "second", "third", "host"):
        s._ctx.profile(mode == "host")
        phi = torch.full_like(rho, 7.0)
        s.solve(rho, phi)
        seen.append((phi, s.last_stats, s.residual_norm()))
    for phi, stats, norm in seen[1:]:
        assert torch.equal(phi, seen[0][0])
        assert stats == seen[0][1] and norm == seen[0][2]


def test_changed_parameters_and_streams(cuda):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    n = 64
    rho = _rho(n, "random")
    s = MultigridPoissonSolver(n, dx=0.5, grav_constant=1.0, tol=1e-3, n_cycles=30)
    ref = {}
    for tol in (1e-3, 1e-8):
        r = MultigridPoissonSolver(n, dx=0.5, grav_constant=1.0, tol=tol, n_cycles=30)
        ref[tol] = torch.empty_like(rho)
        r.solve(rho, ref[tol])
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for k, tol in enumerate((1e-3, 1e-3, 1e-8, 1e-3, 1e-8, 1e-8, 1e-8, 1e-3)):
        s.tol = tol
        with torch.cuda.stream(side if k % 2 else torch.cuda.default_stream()):
            phi = torch.empty_like(rho)
            s.solve(rho, phi)
            assert torch.equal(phi, ref[tol])


def test_engine_steps_and_launch_counts(cuda):
    """An eager engine counts the launches of its graph-run solves as it counts its own."""
    from galaxy_collision_gb300 import ic
    from galaxy_collision_gb300.engine import PMEngine

    icr = ic.plummer(20000, seed=3)
    out = []
    for profiled in (True, False):
        eng = PMEngine(32, 0.75, origin=(-12.0,) * 3, tol=1e-6)
        eng.load(icr.pos, icr.vel, icr.mass, icr.gid)
        eng.ctx.profile(profiled)
        eng.ctx.profile_reset()
        cycles = [eng.prime(0.01).cycles] + [eng.advance(0.01).cycles for _ in range(6)]
        counts = {k: v[0] for k, v in eng.ctx.kernel_stats().items()}
        out.append((cycles, counts, [eng.cur[k].clone() for k in ("x", "vy", "pid")]))
    assert out[0][0] == out[1][0]
    # the graph's loop adds one decision per residual (a reduction kernel)
    extra = out[1][1].pop("reduce") - out[0][1].pop("reduce")
    assert out[0][1] == out[1][1] and 0 <= extra <= sum(out[0][0]) + 7
    for a, b in zip(out[0][2], out[1][2]):
        assert torch.equal(a, b)
