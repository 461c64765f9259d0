"""The binned deposit of particles in no order against the oracle, bit by bit: grids at and
off the tile sizes, an item's and a carry's limits in one tile, particles over the edges,
masses below a quantum, at and beyond the largest a tile sums, and ordered input, which
keeps the ordered kernel."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


def _deposit(pos, mass, G, dx, bits, repeat=1):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    p = ParticleState(len(mass))
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.empty((G, G, G), device="cuda")
    for _ in range(repeat):
        deposit_density(p, rho, dx, fixed_point_bits=bits)
    return rho.cpu().numpy()


@pytest.mark.parametrize("G,dx", [(16, 0.5), (31, 0.3), (33, 1.0), (64, 0.25), (100, 0.3), (117, 1.0)])
@pytest.mark.parametrize("kind", ["uniform", "clustered", "one tile"])
def test_binned_deposit_bit_exact(cuda, G, dx, kind):
    n = max(200_000, G**3 // 8)
    rng = np.random.default_rng(G)
    if kind == "uniform":
        g = rng.uniform(-1.2, G + 0.2, size=(n, 3))
    elif kind == "clustered":
        g = rng.normal(size=(n, 3)) * 0.1 * G + 0.5 * G
    else:  # 8 full items and a remainder, in a few cells of a tile
        g = rng.uniform(0.0, G, size=(n, 3))
        g[: 8 * 8192 + 5] = rng.uniform(9.0, 12.0, size=(8 * 8192 + 5, 3))
        g = g[rng.permutation(n)]
    pos = (g * dx).astype(np.float32)
    mass = (2.0 ** rng.uniform(-30, 0, size=n)).astype(np.float32)
    mass[rng.random(n) < 0.7] = np.float32(1.0 / n)
    want, _, _ = pm.deposit_fixed(pos, mass, dx, G, 52)
    np.testing.assert_array_equal(_deposit(pos, mass, G, dx, 52, repeat=2), want)
    order = np.argsort(pm.cell_keys(pos, dx, G), kind="stable")
    np.testing.assert_array_equal(_deposit(pos[order], mass[order], G, dx, 52), want)


@pytest.mark.parametrize("n,G,dx", [(1_500_000, 100, 0.3), (2_600_000, 64, 0.25)])
def test_blocks_with_several_stretches(cuda, n, G, dx):
    """More particles than one round of blocks copies, and the larger items."""
    rng = np.random.default_rng(n)
    pos = (np.clip(rng.normal(size=(n, 3)) * 0.12, -0.49, 0.49) * G * dx + 0.5 * G * dx).astype(np.float32)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    want, _, _ = pm.deposit_fixed(pos, mass, dx, G, 52)
    np.testing.assert_array_equal(_deposit(pos, mass, G, dx, 52), want)


@pytest.mark.parametrize("bits", [24, 44, 52])
def test_heavy_particles(cuda, bits):
    """Equal masses at the largest sum a tile may hold, and a few beyond it."""
    n, G = 200_000, 32
    rng = np.random.default_rng(bits)
    pos = rng.uniform(0.0, G, size=(n, 3)).astype(np.float32)
    pos[: n // 2] = rng.uniform(3.0, 3.4, size=(n // 2, 3))
    pos = pos[rng.permutation(n)]
    mass = np.full(n, 1.0, np.float32)
    mass[::1000] = 300.0
    want, _, _ = pm.deposit_fixed(pos, mass, 1.0, G, bits)
    np.testing.assert_array_equal(_deposit(pos, mass, G, 1.0, bits), want)


def test_non_finite_positions_are_flagged(cuda):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver
    import ctypes as C

    n, G = 250_000, 32
    ctx = MultigridPoissonSolver(G, dx=1.0, grav_constant=1.0)._ctx
    g = torch.Generator(device="cuda").manual_seed(1)
    pos = [torch.rand(n, device="cuda", generator=g) * G for _ in range(3)]
    m = torch.ones(n, device="cuda")
    rho = torch.empty((G, G, G), device="cuda")

    def flags():
        f = C.c_uint32()
        ctx.call("gc_status", C.byref(f), 1, what="status")
        return f.value

    args = lambda: [p.data_ptr() for p in pos] + [m.data_ptr(), n, 52, rho.data_ptr()]  # noqa: E731
    ctx.call("gc_deposit_cic", *args(), what="deposit")
    assert flags() == 0
    clean = rho.clone()
    pos[1][77_777] = float("nan")
    ctx.call("gc_deposit_cic", *args(), what="deposit")
    assert flags() != 0
    assert not torch.equal(rho, clean) and torch.isfinite(rho).all()
