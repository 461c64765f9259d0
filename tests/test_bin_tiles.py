"""The index arithmetic of the binned deposit (csrc/particles.cu: bin_of, k_bin_count,
k_bin_deposit), restated per axis in float32 and checked on the CPU for every grid it takes:
positions at and next to every cell edge fall in a tile of the grid, their stored copies in
that tile's cells, every corner in its nodes, and the items of any counts fit their array.
On the GPU no index check of the kernels may have failed after deposits of such positions."""

from __future__ import annotations

import numpy as np
import pytest

BIN = (8, 16, 32)  # cells of a tile along x, y, z
MAX_TILES, MAX_GRID = 4096, 256
ITEMS = (8192, 2048)


def _edges(G):
    k = np.arange(-1, G + 1, dtype=np.float32)
    g = np.concatenate([k, np.nextafter(k, np.float32(-9)), np.nextafter(k, np.float32(2 * G + 9)), k + np.float32(0.5)])
    return np.concatenate([g, np.float32([-0.0, -1e-45, 1e-45, 1e-8])])


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_cells_and_corners_lie_in_their_tile(axis):
    B = BIN[axis]
    for G in range(2, MAX_GRID + 1):
        g = _edges(G)
        g = g[(g >= np.float32(-1)) & (g < np.float32(G))]  # what deposits
        tile = np.maximum(np.floor(g).astype(np.int32), 0) // B
        assert tile.min() >= 0 and tile.max() < -(-G // B)
        copy = np.where(g < 0, np.float32(0), g)  # cells -1 leave a massless copy in the first cell
        cell = np.floor(copy).astype(np.int32) - tile * B
        assert cell.min() >= 0 and cell.max() < B  # corner + 1 is one of the B + 1 nodes
    nodes = [b + 1 for b in BIN]
    last = ((BIN[0] - 1 + 1) * nodes[1] + BIN[1] - 1 + 1) * nodes[2] + BIN[2] - 1 + 1
    assert last == nodes[0] * nodes[1] * nodes[2] - 1


def test_tiles_and_items_fit_their_arrays():
    for G in range(2, MAX_GRID + 1):
        assert np.prod([-(-G // b) for b in BIN]) <= MAX_TILES
    rng = np.random.default_rng(1)
    for per in ITEMS:
        for n in (0, 1, per, 200_000, 1 << 25):
            for tiles in (1, 7, MAX_TILES):
                counts = rng.multinomial(n, rng.dirichlet(np.full(tiles, 0.05)))
                assert (-(-counts // per)).sum() <= MAX_TILES + n // per + 1
                assert n + max(ITEMS) < 2**31


@pytest.mark.gpu
@pytest.mark.parametrize("G,dx", [(33, 1.0), (64, 0.3), (117, 0.1)])
def test_no_index_check_fails(cuda, G, dx):
    import torch

    from oracle import pm
    from galaxy_collision_gb300 import _native
    from galaxy_collision_gb300._ops import op_context
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    n = max(200_000, G**3 // 8)
    rng = np.random.default_rng(G)
    pos = (rng.choice(_edges(G).astype(np.float64), size=(n, 3)) * dx).astype(np.float32)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    p = ParticleState(n)
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.empty((G, G, G), device="cuda")
    ctx = op_context(G, dx)
    ctx.status(clear=True)
    deposit_density(p, rho, dx)
    assert ctx.status() & _native.GC_FLAG_INDEX == 0
    np.testing.assert_array_equal(rho.cpu().numpy(), pm.deposit_fixed(pos, mass, dx, G, 52)[0])
