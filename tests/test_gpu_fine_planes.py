"""The finest level as two passes over its planes against one launch per phase on a natural
layout: identical potentials, at grids with partly filled rows, and
strips and stretches of planes that do not divide the grid."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [140, 144, 148, 160, 188, 192, 196, 252, 256])
@pytest.mark.parametrize("plain", [False, True])
def test_planes_bitwise_equal_phases(cuda, n, plain):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    rng = np.random.default_rng(n)
    rho = torch.from_numpy((rng.random((n, n, n)) ** 6).astype(np.float32)).cuda()
    out = []
    for natural in (False, True):
        s = MultigridPoissonSolver(n, dx=0.3, grav_constant=1.0, n_cycles=3, tol=0.0, plain_f32=plain,
                                   natural_layout=natural)
        phi = torch.empty_like(rho)
        s.solve(rho, phi)
        out.append(phi)
    assert torch.equal(out[0], out[1])
