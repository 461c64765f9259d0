"""The standalone gather of many particles in every order a caller may have them (cell order,
drifted from it by up to a cell, none; sparse and dense grids), with particles at and beyond
the grid's edges, against the plain gather in pieces: the same bits."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,dx", [(96, 0.3), (160, 1.0), (220, 0.25)])
@pytest.mark.parametrize("order", ["cells", "drifted", "far drifted", "none"])
def test_gather_orders(cuda, G, dx, order):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.deposit import gather_acceleration

    n, piece = 4_194_304 + 1, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(G)
    r = torch.rand((3, n), device="cuda", generator=g) * (G + 1) - 1.0
    if order != "none":
        c = torch.floor(r).long() + 1
        r = r[:, torch.argsort((c[0] * (G + 2) + c[1]) * (G + 2) + c[2])]
        r += torch.randn((3, n), device="cuda", generator=g) * {"cells": 0.0, "drifted": 0.3, "far drifted": 1.0}[order]
    parts = ParticleState(n)
    field = [torch.randn((G, G, G), device="cuda", generator=g) for _ in range(3)]
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(parts, k).tensor.copy_(r[a] * dx)
    acc = [torch.full((n,), 7.0, device="cuda") for _ in range(3)]
    gather_acceleration(parts, *field, *acc, dx)
    for a in range(0, n, piece):
        b = min(n, a + piece)
        p = ParticleState(b - a)
        for k in ("pos_x", "pos_y", "pos_z"):
            getattr(p, k).tensor.copy_(getattr(parts, k).tensor[a:b])
        want = [torch.full((b - a,), 8.0, device="cuda") for _ in range(3)]
        gather_acceleration(p, *field, *want, dx)
        for u, v in zip(acc, want):
            assert torch.equal(u[a:b], v)
