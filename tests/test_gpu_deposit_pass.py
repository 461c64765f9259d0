"""The deposit where the masses decide between its narrow and its wide pass (mean particles of
2^20 to 2^22 quanta, in cell order): equal masses on either side, masses spread over the limit,
a few heavy ones, none at all, against the oracle bit by bit; and the engine's own deposit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


def _masses(kind, n, rng):
    m = np.full(n, 1.0 / n, np.float32)
    if kind == "spread":
        m *= (2.0 ** rng.uniform(-3, 3, n)).astype(np.float32)
    elif kind == "point":
        m[n // 3] = 0.3
    elif kind == "zero":
        m[:] = 0.0
    elif kind == "heavy half":
        m[n // 2:] *= np.float32(40.0)
    return m


@pytest.mark.parametrize("kind", ["equal", "spread", "point", "zero", "heavy half"])
@pytest.mark.parametrize("n,bits", [(40_000, 36), (40_000, 37), (40_000, 38), (700_001, 40), (700_001, 41), (700_001, 42)])
@pytest.mark.parametrize("dx", [0.25, 0.3])
def test_deposit_bit_exact(cuda, kind, n, bits, dx):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density

    G = 40
    rng = np.random.default_rng(n + bits)
    pos = (rng.normal(size=(n, 3)) * 3.0 * dx + 0.5 * G * dx).astype(np.float32)
    pos = np.ascontiguousarray(pos[np.argsort(pm.cell_keys(pos, dx, G), kind="stable")])
    mass = _masses(kind, n, rng)
    p = ParticleState(n)
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.full((G, G, G), 7.0, device="cuda")
    deposit_density(p, rho, dx, fixed_point_bits=bits)
    np.testing.assert_array_equal(rho.cpu().numpy(), pm.deposit_fixed(pos, mass, dx, G, bits)[0])


@pytest.mark.parametrize("kind", ["equal", "spread"])
def test_engine_states_do_not_depend_on_the_pass(cuda, kind):
    """The same particles in an engine whose quantum puts them at either side of both limits: the
    densities round apart by the quantum alone, far below what moves an f32 position."""
    from galaxy_collision_gb300.engine import PMEngine

    n, G = 300_000, 32
    rng = np.random.default_rng(3)
    pos = (rng.normal(size=(n, 3)) * 3.0).astype(np.float32)
    vel = np.zeros((n, 3), np.float32)
    mass = _masses(kind, n, rng)
    out = []
    for bits in (38, 39, 40, 41, 42):
        eng = PMEngine(G, 1.0, origin=(-16.0,) * 3, tol=1e-6, fixed_point_bits=bits)
        eng.load(pos, vel, mass, np.zeros(n, np.int32))
        eng.prime(0.01)
        for _ in range(3):
            eng.advance(0.01)
        out.append([eng.cur[k].clone() for k in ("x", "y", "z")])
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert float((a - b).abs().max()) < 1e-5
