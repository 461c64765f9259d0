"""The diagnostic reductions against float64 on the host: block remainders, distances on and
beside bin edges, centres that are no f32 values, ranges where the f32 shortcuts do not hold."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _radial(x, m, c, inv_binw, nbins):
    from galaxy_collision_gb300._ops import op_context

    t = [torch.from_numpy(np.ascontiguousarray(x[:, a])).cuda() for a in range(3)] + [torch.from_numpy(m).cuda()]
    hist = torch.empty(nbins, dtype=torch.float64, device="cuda")
    op_context(2, 1.0).call("gc_radial_histogram", *(v.data_ptr() for v in t), len(m), *c, inv_binw, nbins,
                            hist.data_ptr())
    return hist.cpu().numpy()


@pytest.mark.parametrize("n", [1, 255, 4097, 200_003])
@pytest.mark.parametrize("c", [(0.0, 0.0, 0.0), (0.1, -3.3, 31.7)])
@pytest.mark.parametrize("scale", [1.0, 1e-18, 1e17])
def test_radial_histogram_same_bins_as_float64(cuda, n, c, scale):
    rng = np.random.default_rng(n)
    nbins, binw = 64, 0.25 * scale
    x = rng.normal(size=(n, 3)) * 4.0 * scale + np.asarray(c) * scale
    k = n // 3  # on bin edges along an axis, and the neighbouring f32 values
    x[:k] = np.asarray(c) * scale
    x[:k, 0] += binw * rng.integers(0, 70, size=k)
    x = x.astype(np.float32)
    x[:k, 0] = np.nextafter(x[:k, 0], np.float32(np.inf) * rng.choice([-1.0, 1.0], size=k).astype(np.float32)) \
        if n % 2 else x[:k, 0]
    m = (2.0 ** rng.integers(-3, 4, size=n)).astype(np.float32)  # sums are exact
    cs = tuple(v * scale for v in c)
    d = x.astype(np.float64) - np.asarray(cs)
    fb = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]) * (1.0 / binw)
    near = np.abs(fb - np.round(fb)) < 1e-12  # where FMA contraction may decide
    b = np.minimum(fb, nbins - 1).astype(np.int64)
    got = _radial(x[~near], m[~near], cs, 1.0 / binw, nbins)
    np.testing.assert_array_equal(got, np.bincount(b[~near], weights=m[~near].astype(np.float64), minlength=nbins))


@pytest.mark.parametrize("G", [2, 5, 31, 64, 101])
@pytest.mark.parametrize("case", ["mixed", "cancel", "tiny", "zeros"])
def test_grid_energy(cuda, G, case):
    from galaxy_collision_gb300.diagnostics_device import grid_pe_raw

    rng = np.random.default_rng(G)
    a = np.exp(3.0 * rng.normal(size=(G, G, G))).astype(np.float32)
    b = (-rng.random((G, G, G)) - 0.5).astype(np.float32)
    if case == "cancel":
        b *= rng.choice([-1.0, 1.0], size=b.shape).astype(np.float32)
    elif case == "tiny":
        a *= np.float32(1e-25)
        b *= np.float32(1e-12)
    elif case == "zeros":
        a[rng.random(a.shape) < 0.9] = 0.0
    got = grid_pe_raw(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    terms = (a.astype(np.float64) * b.astype(np.float64)).ravel()
    # products are exact in float64; at most G^3 / 16 + 2^12 additions of one thread order
    assert abs(got - math.fsum(terms)) <= np.abs(terms).sum() * 2.0**-53 * 64


@pytest.mark.parametrize("n", [1, 2, 255, 77_825, 311_297, 1_000_003])
def test_particle_sums(cuda, n):
    from galaxy_collision_gb300.data import ParticleState
    from galaxy_collision_gb300.diagnostics_device import particle_scalars

    rng = np.random.default_rng(n)
    x, v = rng.normal(size=(n, 3)).astype(np.float32) * 5 + 30, rng.normal(size=(n, 3)).astype(np.float32)
    m = rng.random(n).astype(np.float32)
    p = ParticleState(n)
    for a, k in enumerate("xyz"):
        getattr(p, "pos_" + k).from_numpy(np.ascontiguousarray(x[:, a].astype(np.float32)))
        getattr(p, "vel_" + k).from_numpy(np.ascontiguousarray(v[:, a]))
    p.mass.from_numpy(m)
    got = particle_scalars(p)
    x, v, m = p_host = (x.astype(np.float32).astype(np.float64), v.astype(np.float64), m.astype(np.float64))
    del p_host
    terms = [m, 0.5 * m * (v * v).sum(1), *(m[:, None] * v).T, *(m[:, None] * np.cross(x, v)).T,
             *(m[:, None] * x).T]
    for g, t in zip(got, terms):
        # pairs of f32: every term and addition to 2^-46 of the running sum
        assert abs(g - math.fsum(t)) <= (np.abs(t).sum() + 90.0 * np.abs(m).sum()) * 2.0**-46 + 1e-300
