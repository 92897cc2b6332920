"""Calls with a handful of tokens: what a launch prepares once per call must not fall to the few blocks that have tiles."""

import statistics

import pytest
import torch

import miniworld_b200 as mw

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _module(kind):
    g = torch.Generator().manual_seed(7)
    m = {"out": lambda: mw.TriangleMultiplication(128, 128, outgoing=True),
         "bidir": lambda: mw.BidirectionalTriangleMultiplication(128, 128),
         "narrow": lambda: mw.TriangleMultiplication(64, 128, outgoing=False)}[kind]()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_((1.0 if p.dim() == 1 else 0.0) + torch.randn(p.shape, generator=g) * (0.1 if p.dim() == 1 else p.shape[-1] ** -0.5))
    return m.to(DEV).to(torch.bfloat16).eval()


def _device_us(m, n, calls=20):
    """Device time of a call: replays of a graph of ``calls`` calls (no host work between the launches)."""
    c = m.d_pair
    z = torch.randn(1, n, n, c, generator=torch.Generator().manual_seed(n)).to(torch.bfloat16).to(DEV)
    with torch.no_grad():
        m(z)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(calls):
                m(z)
    graph.replay()
    times = []
    for _ in range(9):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end) * 1e3 / calls)
    return statistics.median(times)


@pytest.mark.parametrize("kind", ["out", "bidir", "narrow"])
def test_fewer_tokens_take_no_longer(kind):
    """N = 1 has one tile where N = 64 has 64, each of which takes one pair of CTAs: no more work and no longer a chain. (20 % for
    the spread of medians of some 15 us.)"""
    m = _module(kind)
    reference = _device_us(m, 64)
    times = {n: _device_us(m, n) for n in (1, 2, 5, 8, 16, 32)}
    assert all(t <= 1.2 * reference for t in times.values()), (reference, times)
