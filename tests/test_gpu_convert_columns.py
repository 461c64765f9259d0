"""Density and moments from the fixed-point grid, columns gathered in batches of 8, 16 and 32.

Grids at the lines between the batch sizes, with a last batch that is not full and with
columns beyond one stretch of 256 nodes; clustered particles leave most columns empty.
The density is the exact fixed-point sum rounded once: equal to the oracle's. The moments
show in the multipole faces, which the solver also forms from the density (FP32
compensated sums, 3 * 2^-24 of each moment; the quadrupole's share of the potential is
below (G/d)^2 = 16 times that, with the distance d at least G/4)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import pm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [8, 33, 49, 50, 69, 70, 100, 257])
@pytest.mark.parametrize("spread", [0.9, 0.2])
def test_density_and_faces(cuda, G, spread):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import deposit_density
    from galaxy_collision_gb300.engine import PMEngine
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    n = 3000
    rng = np.random.default_rng(G)
    pos = ((G - 1) * (0.5 + spread * (rng.random((n, 3)) - 0.5))).astype(np.float32)
    mass = rng.uniform(0.2, 1.0, n).astype(np.float32)
    p = ParticleState(n)
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(p, k).from_numpy(np.ascontiguousarray(pos[:, a]))
    p.mass.from_numpy(mass)
    rho = torch.empty((G, G, G), device="cuda")
    deposit_density(p, rho, 1.0, fixed_point_bits=44)
    want, _, _ = pm.deposit_fixed(pos, mass, 1.0, G, 44)
    np.testing.assert_array_equal(rho.cpu().numpy(), want)

    eng = PMEngine(G, 1.0, tol=1e-3, max_cycles=1, sort_every=0, fixed_point_bits=44)
    eng.load(pos, np.zeros((n, 3), np.float32), mass)
    eng.prime(0.01)
    got = eng.potential()
    s = MultigridPoissonSolver(G, dx=1.0, grav_constant=1.0, tol=1e-3, n_cycles=1)
    phi = torch.empty_like(rho)
    s.solve(rho, phi)
    for a in range(3):
        for e in (0, G - 1):
            f, g = got.select(a, e).double(), phi.select(a, e).double()
            assert float(((f - g).abs() / g.abs()).max()) <= 2.0**-24 * 2 * 3 * 17
