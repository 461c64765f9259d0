"""Kick and drift on four particles a thread: remainders of four, and arrays off the 16-byte
boundary (one particle a thread) against the same FP32 operations, bit by bit."""

from __future__ import annotations

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 1024, 4097])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("name", ["gc_kick", "gc_drift"])
def test_kick_drift_bits(cuda, n, shift, name):
    from galaxy_collision_gb300.solver.multigrid import MultigridPoissonSolver

    ctx = MultigridPoissonSolver(8, dx=1.0, grav_constant=1.0)._ctx
    g = torch.Generator(device="cuda").manual_seed(n)
    buf = [torch.randn(n + 9, device="cuda", generator=g) for _ in range(6)]
    want = [b.clone() for b in buf]
    dt = 0.37
    for k in range(3):
        want[k][shift:shift + n] += buf[3 + k][shift:shift + n] * torch.tensor(dt, device="cuda")
    ctx.call(name, *[b[shift:].data_ptr() for b in buf], n, C.c_float(dt), what=name)
    torch.cuda.synchronize()
    for b, w in zip(buf, want):
        assert torch.equal(b, w)
