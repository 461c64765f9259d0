"""The grid energy's sum of products over the range of f32 against 64 bits: products that
underflow, overflow or mix with ordinary ones, zeros, and infinities."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 64])
@pytest.mark.parametrize("sa,sb", [(1.0, 1.0), (1e-20, 1e-15), (1e-30, 1e-12), (3e-39, 2e-39), (1e20, 1e15), (1e37, 1e30),
                                   (1e-37, 1e37), (1e37, 3e-39)])
@pytest.mark.parametrize("mix", ["even", "zeros", "wide", "one large", "apart"])
def test_sum_of_products(cuda, n, sa, sb, mix):
    """The three parts keep 2^-70 of the largest product; adding them and the threads' sums in FP64
    leaves 2^-53 for each of some ten additions, of the sum of the products' magnitudes."""
    from galaxy_collision_gb300.diagnostics_device import grid_pe_raw

    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.rand((n, n, n), device="cuda", generator=g, dtype=torch.float64) + 0.5
    b = torch.randn((n, n, n), device="cuda", generator=g, dtype=torch.float64)
    if mix == "zeros":
        a[torch.rand((n, n, n), device="cuda", generator=g) < 0.7] = 0.0
    elif mix == "wide":
        a *= 10.0 ** (-30.0 * torch.rand((n, n, n), device="cuda", generator=g, dtype=torch.float64))
    elif mix == "one large":
        a *= 1e-25
        a[n // 2, 3, 5] = 1.0
    elif mix == "apart":  # where one factor is large the other is not there
        pick = torch.rand((n, n, n), device="cuda", generator=g) < 0.5
        a[pick] = 0.0
        b[~pick] *= 1e-25
    a, b = (a * sa).float(), (b * sb).float()
    p = a.double() * b.double()
    got = grid_pe_raw(a, b)
    assert abs(got - float(p.sum())) <= 16 * 2.0**-53 * float(p.abs().sum())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_values_come_through(cuda, value):
    from galaxy_collision_gb300.diagnostics_device import grid_pe_raw

    a, b = torch.ones((20, 20, 20), device="cuda"), torch.ones((20, 20, 20), device="cuda")
    a[3, 4, 5] = value
    got = grid_pe_raw(a, b)
    assert np.isinf(got) if np.isinf(value) else np.isnan(got)
    b[3, 4, 5] = 0.0
    assert np.isnan(grid_pe_raw(a, b))
