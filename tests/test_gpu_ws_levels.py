"""The network's passes between its levels, on sizes where their lines have remainders.

A thread of the upsampling and of the pool's adjoint takes four children of a parent, 64
threads a block along the line: lines below one block (24, and 12 and 6 on the levels
below) and lines of a block and a part of one (72). Tolerances as for the other sizes:
bf16 activations, whose roundings flip between fp32 and fp64 accumulation, 1 % over the
prediction and 2 % over the gradient."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import warmstart as ows

pytestmark = pytest.mark.gpu


def _inputs(R):
    rng = np.random.default_rng(R)
    p = []
    for ci, co, _, _ in ows.LAYERS:
        p += [rng.normal(0.0, np.sqrt(2.0 / (27 * ci)), size=27 * co * ci), rng.normal(0.0, 0.05, size=co)]
    feat = rng.normal(size=(4, R, R, R)).astype(np.float16)
    target = (0.1 * rng.normal(size=(R, R, R))).astype(np.float16)
    return np.concatenate(p).astype(np.float32), feat, target


@pytest.mark.parametrize("R,grad", [(24, True), (72, False)])
def test_levels_with_remainders(cuda, R, grad):
    from galaxy_collision_gb300.warmstart import WarmStartNet

    p, feat, target = _inputs(R)
    f, t = torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda()
    net = WarmStartNet(R, params=p)
    y = net.forward(f).cpu().numpy()
    net.backward(t)
    g = net.grads().cpu().numpy()
    assert net.status() == 0
    yo, cache = ows.forward(p, feat, emulate=True)
    assert rel_l2(y, yo) < 1e-2
    if grad:
        _, go = ows.backward(cache, target.astype(np.float64), emulate=True)
        assert rel_l2(g, go) < 2e-2
