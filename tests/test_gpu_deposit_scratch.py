"""The scratch of the standalone deposit of particles in no order: a deposit recorded in a CUDA
graph after an eager one keeps its density when a larger eager deposit of the same grid
has been made since, the scratch is bounded whatever the particle count, and more particles
than the passes take at a time are summed as few are."""

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


def test_scratch_is_bounded_and_given_back(cuda):
    from galaxy_collision_gb300._ops import clear_cache
    from galaxy_collision_gb300.deposit import deposit_density

    G, n = 32, 60_000_000
    p = _parts(n, G, 3)
    rho = torch.empty((G, G, G), device="cuda")
    clear_cache()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    deposit_density(p, rho, 1.0)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 800_000_000  # 671 MB and the context, not 20 bytes a particle
    clear_cache()
    assert free - torch.cuda.mem_get_info()[0] < 40_000_000


def test_more_particles_than_a_pass_takes(cuda):
    from galaxy_collision_gb300.deposit import deposit_density

    G, n = 40, (1 << 25) + 300_001
    p = _parts(n, G, 4, dx=0.3)
    rho = torch.empty((G, G, G), device="cuda")
    deposit_density(p, rho, 0.3)
    assert torch.equal(rho.cpu(), _want(p, G, 0.3))


def test_the_most_particles_a_call_takes(cuda):
    """2^31 - 1 of them: as the sum of two deposits of halves, whose sums round apart only in
    the f32 density (three roundings of 2^-24, and weights that are the same)."""
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    G, n = 32, 2**31 - 1
    g = torch.Generator(device="cuda").manual_seed(6)
    arr = {k: torch.empty(n, device="cuda") for k in ("pos_x", "pos_y", "pos_z", "mass")}
    for k, a in arr.items():
        for part in a.split(1 << 28):
            part.uniform_(0.0 if k != "mass" else 0.5, G - 1.0 if k != "mass" else 1.5, generator=g)

    class View:
        def __init__(self, lo, hi):
            self.n = hi - lo
            for k, a in arr.items():
                setattr(self, k, a[lo:hi])

    rho = [torch.empty((G, G, G), device="cuda") for _ in range(3)]
    half = 1 << 30
    for r, (lo, hi) in zip(rho, ((0, n), (0, half), (half, n))):
        deposit_density(View(lo, hi), r, 1.0)
    total = rho[1].double() + rho[2].double()
    assert float(((rho[0].double() - total).abs() / total).max()) < 4 * 2.0**-24
    del arr
    torch.cuda.empty_cache()
