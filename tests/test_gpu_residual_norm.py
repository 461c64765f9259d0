"""The residual's norm and the verdict from the block partials: one block over up to 4096
partials, chunks first above that.

Sizes with one partial, a few, around 256 and 4096, and 16 thousand; the natural layout
sums the same residual over other blocks. A block adds at most 1024 squares in FP32, so
the two norms agree to 2^-20."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 9, 34, 48, 64, 66, 128, 129, 180, 256])
def test_norm_of_one_cycle_against_the_natural_layout(cuda, n):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    g = torch.Generator(device="cuda").manual_seed(n)
    rho = torch.rand((n, n, n), device="cuda", generator=g) ** 3
    stats = []
    for kw in ({}, dict(natural_layout=True)):
        s = MultigridPoissonSolver(n, dx=0.5, grav_constant=1.0, tol=0.0, n_cycles=1, **kw)
        for _ in range(3):  # host loop, then the device's
            phi = torch.empty_like(rho)
            s.solve(rho, phi)
            stats.append(s.last_stats)
    res = [st["res_norm"] for st in stats]
    assert res[0] > 0.0 or n < 16
    assert res[0] == res[1] == res[2] and res[3] == res[4] == res[5]
    assert abs(res[0] - res[3]) <= 2.0**-20 * res[0]
