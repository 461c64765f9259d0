"""The standalone deposit of as few particles as the binned passes take, in every order a caller
may have them (cell order, drifted from it, none), on grids of the most tiles and with partial
last tiles, against the oracle bit by bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,dx", [(130, 0.3), (201, 1.0), (256, 0.25)])
@pytest.mark.parametrize("order", ["cells", "drifted", "far drifted", "none"])
def test_deposit_orders(cuda, G, dx, order):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    n = G**3 // 8 + 1
    rng = np.random.default_rng(G)
    pos = (rng.uniform(-1.0, G, size=(n, 3)) * dx).astype(np.float32)
    if order != "none":
        pos = pos[np.argsort(pm.cell_keys(pos, dx, G), kind="stable")]
        pos += rng.normal(size=(n, 3)).astype(np.float32) * np.float32(dx * {"cells": 0.0, "drifted": 0.3, "far drifted": 1.0}[order])
    pos = np.ascontiguousarray(pos)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    p = ParticleState(n)
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.full((G, G, G), 7.0, device="cuda")
    deposit_density(p, rho, dx)
    np.testing.assert_array_equal(rho.cpu().numpy(), pm.deposit_fixed(pos, mass, dx, G, 52)[0])
