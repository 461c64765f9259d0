"""The sorted deposit's fine-quantum pass against the oracle: the corner split h 2^20 + l at
its limits (2^22, 2^41 quanta), few and many particles, boxes that do and do not fit a warp."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


def _deposit(pos, mass, G, dx, bits):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    p = ParticleState(len(mass))
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.empty((G, G, G), device="cuda")
    deposit_density(p, rho, dx, fixed_point_bits=bits)
    return rho.cpu().numpy()


@pytest.mark.parametrize("n", [1, 255, 257, 5000, 400_003])
@pytest.mark.parametrize("bits,dx", [(52, 0.25), (52, 0.3), (44, 0.25), (40, 0.3)])
@pytest.mark.parametrize("ordered", [True, False])
def test_deposit_bit_exact(cuda, n, bits, dx, ordered):
    G = 32
    rng = np.random.default_rng(n + bits)
    pos = (rng.normal(size=(n, 3)) * 1.5 * dx + 0.5 * G * dx).astype(np.float32)
    pos[::7] = rng.uniform(-1.5 * dx, (G + 0.5) * dx, size=pos[::7].shape)  # sparse, and over the edges
    # masses over 2^30: below one quantum, below and above both limits of the passes
    mass = (2.0 ** rng.uniform(-30, 0, size=n)).astype(np.float32)
    mass[rng.random(n) < 0.5] = np.float32(1.0 / n)
    if ordered:
        order = np.argsort(pm.cell_keys(pos, dx, G), kind="stable")
        pos, mass = np.ascontiguousarray(pos[order]), mass[order]
    want, _, _ = pm.deposit_fixed(pos, mass, dx, G, bits)
    np.testing.assert_array_equal(_deposit(pos, mass, G, dx, bits), want)
