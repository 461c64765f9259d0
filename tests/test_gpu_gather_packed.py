"""The gather of many particles, in no order (packed fields) and in the order of their cells
(three fields), against the plain gather in pieces too small for either: the same bits,
at the grid's edges and outside it too."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,dx", [(2, 1.0), (33, 0.3), (128, 0.25)])
@pytest.mark.parametrize("ordered", [False, True])
def test_gather_bits(cuda, G, dx, ordered):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    n, piece = 4_194_304 + 77, 1_000_003
    ctx = MultigridPoissonSolver(G, dx=dx, grav_constant=1.0)._ctx
    g = torch.Generator(device="cuda").manual_seed(G)
    r = (torch.rand((3, n), device="cuda", generator=g) * (G + 2) - 1.5) * dx
    if ordered:
        c = torch.floor(r / dx).clamp(-1, G).long() + 1
        r = r[:, torch.argsort((c[0] * (G + 2) + c[1]) * (G + 2) + c[2])]
    r[:, 5] = float("nan")
    pos = [r[a].contiguous() for a in range(3)]
    field = [torch.randn(G**3, device="cuda", generator=g) for _ in range(3)]
    acc = [torch.full((n,), 7.0, device="cuda") for _ in range(3)]
    want = [torch.full((n,), 8.0, device="cuda") for _ in range(3)]
    args = [t.data_ptr() for t in field]
    for _ in range(2):
        ctx.call("gc_gather_accel", *[t.data_ptr() for t in pos], n, *args, *[t.data_ptr() for t in acc], what="gather")
    for a in range(0, n, piece):
        b = min(n, a + piece)
        ctx.call("gc_gather_accel", *[t[a:].data_ptr() for t in pos], b - a, *args, *[t[a:].data_ptr() for t in want],
                 what="gather")
    for u, v in zip(acc, want):
        assert torch.equal(u, v)
