"""Gathers of many particles on two streams at once over the same grid: different fields and
particles, one set in no order and one in the order of its cells, against the plain gather in
pieces; and one recorded in a CUDA graph, replayed beside eager ones."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

N, G, DX, PIECE = 4_194_304 + 77, 96, 0.5, 1_000_003


def _set(seed, ordered):
    from galaxy_collision_gb300.data import ParticleState

    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand((3, N), device="cuda", generator=g) * (G - 1)
    if ordered:
        c = torch.floor(r).long()
        r = r[:, torch.argsort((c[0] * G + c[1]) * G + c[2])]
    parts = ParticleState(N)
    for a, k in enumerate(("pos_x", "pos_y", "pos_z")):
        getattr(parts, k).tensor.copy_(r[a] * DX)
    return parts, [torch.randn((G, G, G), device="cuda", generator=g) for _ in range(3)]


def _gather(parts, field, acc):
    from galaxy_collision_gb300.deposit import gather_acceleration

    gather_acceleration(parts, *field, *acc, DX)


def _want(parts, field):
    from galaxy_collision_gb300.data import ParticleState

    want = [torch.empty(N, device="cuda") for _ in range(3)]
    for a in range(0, N, PIECE):
        b = min(N, a + PIECE)
        p = ParticleState(b - a)
        for k in ("pos_x", "pos_y", "pos_z"):
            getattr(p, k).tensor.copy_(getattr(parts, k).tensor[a:b])
        acc = [torch.empty(b - a, device="cuda") for _ in range(3)]
        _gather(p, field, acc)
        for w, v in zip(want, acc):
            w[a:b] = v
    return want


@pytest.mark.parametrize("ordered", [(False, False), (False, True)])
def test_two_streams(cuda, ordered):
    sets = [_set(5 + k, o) for k, o in enumerate(ordered)]
    want = [_want(*s) for s in sets]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    rounds = 6
    acc = [[[torch.full((N,), 7.0, device="cuda") for _ in range(3)] for _ in range(rounds)] for _ in sets]
    torch.cuda.synchronize()
    for r in range(rounds):
        for k, st in enumerate(streams):
            with torch.cuda.stream(st):
                _gather(*sets[k], acc[k][r])
    torch.cuda.synchronize()
    for k in range(2):
        for r in range(rounds):
            for u, v in zip(acc[k][r], want[k]):
                assert torch.equal(u, v)


def test_recorded_gather_beside_eager_ones(cuda):
    sets = [_set(5 + k, False) for k in range(2)]
    want = [_want(*s) for s in sets]
    acc = [[torch.empty(N, device="cuda") for _ in range(3)] for _ in sets]
    _gather(*sets[1], acc[1])  # an eager gather first: whatever it leaves behind is there for the recording
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _gather(*sets[0], acc[0])
    other = torch.cuda.Stream()
    for r in range(4):
        for a in acc[0] + acc[1]:
            a.fill_(7.0)
        torch.cuda.synchronize()
        graph.replay()
        with torch.cuda.stream(other):
            _gather(*sets[1], acc[1])
        torch.cuda.synchronize()
        for k in range(2):
            for u, v in zip(acc[k], want[k]):
                assert torch.equal(u, v)
