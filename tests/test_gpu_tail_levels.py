"""The single-CTA tail with one to four levels of every size it can have, against the exact
solution of the discrete problem (sine transforms in float64)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import dst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [4, 5, 6, 8, 9, 10, 13, 16, 17, 18, 21, 25, 30, 32, 33, 34, 47])
def test_solution_and_convergence(cuda, G):
    from galaxy_collision_gb300.solver import make_solver

    rng = np.random.default_rng(G)
    rho = (rng.random((G, G, G)) ** 3).astype(np.float32)
    want = dst.solve_reference_problem(rho, 0.5, 1.0)
    solver = make_solver("multigrid", G, dx=0.5, grav_constant=1.0, tol=1e-9, n_cycles=20)
    phi = torch.empty((G, G, G), device="cuda")
    solver.solve(torch.from_numpy(rho).cuda(), phi)
    # a cycle contracts by 0.1 to 0.2, so 1e-9 takes 10 to 14 of them from a cold start
    assert solver.last_stats["converged"] and solver.last_cycles <= 14
    # f32 rounding of the result (2^-24) and the residual's 1e-9 times the condition
    # number of the 7-point problem, at most 0.41 G^2
    err = np.linalg.norm(phi.cpu().numpy() - want) / np.linalg.norm(want)
    assert err <= 2.0**-23 + 1e-9 * G * G
