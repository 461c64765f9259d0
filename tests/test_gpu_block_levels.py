"""The block kernels (a level's way down and way up in one launch each) against one launch
per phase on a natural layout: identical potentials, at grids around the blocks' sizes, for
every sweep count they are built for and for the ones that fall back."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [18, 24, 25, 33, 34, 50, 64, 71, 97, 98, 128, 129, 132, 161])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 1), (1, 2), (2, 1), (3, 2), (2, 0)])
@pytest.mark.parametrize("plain", [False, True])
def test_blocks_bitwise_equal_phases(cuda, n, pre, post, plain):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    rng = np.random.default_rng(n)
    rho = torch.from_numpy((rng.random((n, n, n)) ** 6).astype(np.float32)).cuda()
    out = []
    for natural in (False, True):
        s = MultigridPoissonSolver(n, dx=0.3, grav_constant=1.0, n_cycles=3, tol=0.0, pre_sweeps=pre, post_sweeps=post,
                                   plain_f32=plain, natural_layout=natural)
        phi = torch.empty_like(rho)
        s.solve(rho, phi)
        out.append(phi)
    assert torch.equal(out[0], out[1])
