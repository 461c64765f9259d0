"""The one-pass right-hand side and moments of a density (the standalone solve's first
kernel) against NumPy in float64: grids below, at and off its unit of eight columns and
its 32-node loads."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [2, 3, 7, 8, 9, 31, 33, 64, 97])
def test_moments_and_rhs_norm(cuda, G):
    from galaxy_collision_gb300.solver import make_solver

    dx, grav = 0.375, 1.3
    rng = np.random.default_rng(G)
    rho = (rng.random((G, G, G)) ** 4 * 3.0).astype(np.float32)
    solver = make_solver("multigrid", G, dx=dx, grav_constant=grav, tol=1e-3)
    dev = torch.from_numpy(rho).cuda()
    got = np.array(solver.moments(dev))
    m = rho.astype(np.float64) * dx**3
    x = np.arange(G) * dx
    want = np.array([m.sum()] + [np.einsum(e, m, x) for e in ("ijk,i->", "ijk,j->", "ijk,k->")]
                    + [np.einsum(e, m, x * x) for e in ("ijk,i->", "ijk,j->", "ijk,k->")]
                    + [np.einsum(e, m, x, x) for e in ("ijk,i,j->", "ijk,i,k->", "ijk,j,k->")])
    # every term is non-negative and carries at most two f32 product roundings (2^-24
    # each); the compensated sums add less than one more
    assert np.all(np.abs(got - want) <= 3.0 * 2.0**-24 * want)
    phi = torch.zeros_like(dev)
    solver.solve(dev, phi)
    norm = 4.0 * np.pi * grav * np.sqrt((rho.astype(np.float64) ** 2).sum())
    # f32 squares and per-thread f32 sums of at most G^3 / 2 terms of one sign
    assert abs(solver.last_stats["rhs_norm"] - norm) <= norm * 2.0**-24 * (8 + G)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_density_is_refused(cuda, bad):
    from galaxy_collision_gb300._native import GCError
    from galaxy_collision_gb300.solver import make_solver

    rho = torch.ones((17, 17, 17), device="cuda")
    rho[16, 9, 5] = bad
    solver = make_solver("multigrid", 17, dx=1.0, grav_constant=1.0)
    with pytest.raises(GCError, match="non-finite"):
        solver.solve(rho, torch.zeros_like(rho))
