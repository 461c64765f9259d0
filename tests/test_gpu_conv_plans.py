"""Every tile plan of the warm-start convolutions gives the same bits.

The marching strips, the blocks of whole lines and every split of the output channels
accumulate an output in the same order, so the prediction and the data gradients do not
depend on the plan. Sizes: one strip of 8-voxel tiles (16), a width that no power of two
above 16 divides (48), lines whose halo is just inside (112) and beyond (128) what a
block's tensor-map box may span, and levels whose size is not a multiple of a strip's
lines (24, 40: blocks only)."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(R, seed):
    from galaxy_collision_gb300.warmstart import WarmStartNet, layer_table

    rng = np.random.default_rng(seed)
    p = []
    for ci, co, _, _ in layer_table():
        p += [rng.normal(0.0, np.sqrt(2.0 / (27 * ci)), size=27 * co * ci), rng.normal(0.0, 0.05, size=co)]
    return WarmStartNet(R, params=np.concatenate(p).astype(np.float32))


def _set(net, layer, kind, index):
    n = C.c_int()
    rc = net._lib.gc_ws_set_plan(net._h, layer, kind, index, C.cast(C.byref(n), C.c_void_p))
    assert rc == 0
    return n.value


def _run(net, feat, target):
    y = net.forward(feat).clone()
    net.backward(target)
    g = net.grads().clone()
    assert net.status() == 0
    return y, g


@pytest.mark.parametrize("R", [16, 24, 32, 40, 48, 64, 112, 128])
def test_convolution_bits_do_not_depend_on_the_plan(cuda, R):
    net = _net(R, R)
    gen = torch.Generator(device="cuda").manual_seed(R)
    feat = torch.randn((4, R, R, R), device="cuda", generator=gen).half()
    target = torch.randn((R, R, R), device="cuda", generator=gen).half()
    counts = {(l, k): _set(net, l, k, -1) for l in range(11) for k in (0, 1)}
    for (l, k), n in counts.items():  # the first candidate is a block with unsplit channels
        _set(net, l, k, 0)
    y0, g0 = _run(net, feat, target)
    assert torch.isfinite(y0).all() and float(y0.abs().max()) > 0.0
    most = max(counts.values())
    step = 1 if R <= 48 else 5  # all of them at the small sizes; 5 is coprime to the nesting of the enumeration
    for i in range(1, most, step):
        for (l, k), n in counts.items():
            _set(net, l, k, i % n)
        y, g = _run(net, feat, target)
        assert torch.equal(y, y0), i
        assert torch.equal(g, g0), i
