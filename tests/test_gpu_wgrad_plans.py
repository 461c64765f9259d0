"""The warm-start network's weight gradient under every plan, and against the oracle.

Plans change the blocks of voxels, how many partial sums they are dealt to, and with them
how the taps are divided, the ring's depth and how often a CTA meets another block. All
of them add the same products in FP32, in another order: over n voxels the sums differ by
about 2^-24 sqrt(n) of their size, and 2^-21 sqrt(n) in the 2-norm of a layer is
allowed. 24 and 40 have levels of 12, 6, 3 and 20, 10, 5 voxels.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import warmstart as ows

pytestmark = pytest.mark.gpu


def _params(seed):
    rng = np.random.default_rng(seed)
    p = []
    for ci, co, _, _ in ows.LAYERS:
        p += [rng.normal(0.0, np.sqrt(2.0 / (27 * ci)), size=27 * co * ci), rng.normal(0.0, 0.05, size=co)]
    return np.concatenate(p).astype(np.float32)


def _set(net, layer, index):
    n = C.c_int()
    assert net._lib.gc_ws_set_plan(net._h, layer, 2, index, C.cast(C.byref(n), C.c_void_p)) == 0
    return n.value


@pytest.mark.parametrize("R", [16, 24, 48, 64])
def test_weight_gradient_does_not_depend_on_the_plan(cuda, R):
    from galaxy_collision_gb300.warmstart import WarmStartNet, param_slices

    net = WarmStartNet(R, params=_params(R))
    gen = torch.Generator(device="cuda").manual_seed(R)
    feat = torch.randn((4, R, R, R), device="cuda", generator=gen).half()
    target = torch.randn((R, R, R), device="cuda", generator=gen).half()
    net.forward(feat)
    counts = [_set(net, l, -1) for l in range(11)]
    tol = 2.0**-21 * R**1.5
    base = None
    for i in range(max(counts)):
        for l, n in enumerate(counts):
            _set(net, l, i % n)
        net.backward(target)
        g = net.grads().double()
        assert net.status() == 0
        if base is None:
            base = g
            continue
        for l, (w, b) in enumerate(param_slices()):
            for sl in (w, b):
                assert float((g[sl] - base[sl]).norm()) <= tol * float(base[sl].norm()), (i, l)


@pytest.mark.parametrize("R", [24, 40])
def test_weight_gradient_matches_oracle(cuda, R):
    from galaxy_collision_gb300.warmstart import WarmStartNet, param_slices

    p = _params(R + 1)
    rng = np.random.default_rng(R)
    feat = rng.normal(size=(4, R, R, R)).astype(np.float16)
    target = (0.1 * rng.normal(size=(R, R, R))).astype(np.float16)
    net = WarmStartNet(R, params=p)
    net.forward(torch.from_numpy(feat).cuda())
    net.backward(torch.from_numpy(target).cuda())
    g = net.grads().cpu().numpy()
    assert net.status() == 0
    _, cache = ows.forward(p, feat, emulate=True)
    _, go = ows.backward(cache, target.astype(np.float64), emulate=True)
    # bf16 resolution, as for the whole backward pass elsewhere
    assert rel_l2(g, go) < 2e-2
    for l, (w, b) in enumerate(param_slices()):
        assert rel_l2(g[w], go[w]) < 6e-2, l
        assert rel_l2(g[b], go[b]) < 6e-2, l
