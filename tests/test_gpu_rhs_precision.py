"""The right-hand side's norm and the moments of a density against 64 bits, where one pass makes
both (the norms and column sums of whole grids, not of samples)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 64, 97, 128, 200, 256])
@pytest.mark.parametrize("power", [1, 5])
def test_norm_and_moments(cuda, n, power):
    """b is rounded to f32 as the kernel rounds it. Eight squares are summed by a tree, within
    4 * 2^-24 of their sum, and these sums as pairs: the errors of n^3 / 8 of them, of either
    sign, add up to 2^-22 / sqrt(n^3 / 8), half of that in the root; ten times that is asked for.
    The moments' Kahan sums leave second-order terms of each column: they agree to 1e-8."""
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    dx = 0.5
    g = torch.Generator(device="cuda").manual_seed(n + power)
    rho = torch.rand((n, n, n), device="cuda", generator=g) ** power
    s = MultigridPoissonSolver(n, dx=dx, grav_constant=1.0, n_cycles=1, tol=0.0)
    phi = torch.empty_like(rho)
    s.solve(rho, phi)
    b = (torch.tensor(4.0 * np.pi, dtype=torch.float32, device="cuda") * rho) * torch.tensor(dx * dx, dtype=torch.float32)
    want = float(b.double().square().sum().sqrt()) / (dx * dx)
    assert abs(s.last_stats["rhs_norm"] / want - 1.0) < 10.0 * 2.0**-23 / np.sqrt(n**3 / 8.0)
    t = torch.arange(n, dtype=torch.float64, device="cuda") * dx
    r = rho.double() * dx**3
    c = [r.sum((1, 2)), r.sum((0, 2)), r.sum((0, 1))]
    exact = [r.sum()] + [(q * t).sum() for q in c] + [(q * t * t).sum() for q in c]
    exact += [(r.sum(k) * t[:, None] * t[None, :]).sum() for k in (2, 1, 0)]
    for a, e in zip(s.moments(rho), exact):
        assert abs(a / float(e) - 1.0) < 1e-8


def test_overflow_of_the_norm_stays_an_infinity(cuda):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    n = 32
    rho = torch.full((n, n, n), 1e25, device="cuda")
    s = MultigridPoissonSolver(n, dx=1.0, grav_constant=1.0, n_cycles=1, tol=0.0)
    s.solve(rho, torch.empty_like(rho))
    assert s.last_stats["rhs_norm"] == float("inf")
