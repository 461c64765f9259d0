"""The scratch of the standalone deposit of particles in no order: a deposit recorded in a CUDA
graph after an eager one keeps its density when a larger eager deposit of the same grid
has been made since."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


def _parts(n, G, seed, dx=1.0):
    from galaxy_collision_gb300.data import ParticleState

    g = torch.Generator(device="cuda").manual_seed(seed)
    p = ParticleState(n)
    for k in ("pos_x", "pos_y", "pos_z"):
        getattr(p, k).tensor.copy_(torch.rand(n, device="cuda", generator=g) * (G * dx))
    p.mass.tensor.copy_(torch.rand(n, device="cuda", generator=g) + 0.5)
    return p


def _want(p, G, dx=1.0):
    pos = np.stack([getattr(p, k).tensor.cpu().numpy() for k in ("pos_x", "pos_y", "pos_z")], 1)
    return torch.from_numpy(pm.deposit_fixed(pos, p.mass.tensor.cpu().numpy(), dx, G, 52)[0])


def test_recorded_deposit_outlives_a_larger_eager_one(cuda):
    from galaxy_collision_gb300.deposit import deposit_density

    G = 48
    few, many = _parts(250_000, G, 1), _parts(1_500_000, G, 2)
    rho = [torch.empty((G, G, G), device="cuda") for _ in range(2)]
    want = [_want(few, G), _want(many, G)]
    deposit_density(few, rho[0], 1.0)
    assert torch.equal(rho[0].cpu(), want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        deposit_density(few, rho[0], 1.0)
    for _ in range(2):
        deposit_density(many, rho[1], 1.0)
        torch.cuda.synchronize()
        rho[0].fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(rho[0].cpu(), want[0]) and torch.equal(rho[1].cpu(), want[1])
