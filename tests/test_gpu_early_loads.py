"""The prologue and the epilogues read z (the epilogues also the packed weights) while the kernel before them finishes. What a
call is given may have been written by the launch right before the call: stacks of calls, each on the output of the one before,
against the same calls with the device idle in between. The sizes give a CTA no, one, two and more tiles."""

import pytest
import torch

import miniworld_b200 as mw

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KINDS = {
    "outgoing": lambda c: mw.TriangleMultiplication(c, 128, outgoing=True),
    "incoming": lambda c: mw.TriangleMultiplication(c, 128, outgoing=False),
    "bidirectional": lambda c: mw.BidirectionalTriangleMultiplication(c, 128 if c == 128 else 64),
}


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("kind,c", [("outgoing", 128), ("incoming", 64), ("bidirectional", 128), ("bidirectional", 64)])
@pytest.mark.parametrize("n", [8, 72, 144, 203, 296])
def test_stack_of_calls(kind, c, n, graph):
    g = torch.Generator().manual_seed(n)
    modules = [KINDS[kind](c).to(DEV).to(torch.bfloat16).eval() for _ in range(2)]
    with torch.no_grad():
        for m in modules:
            for p in m.parameters():
                p.copy_((1.0 if p.dim() == 1 else 0.0) + torch.randn(p.shape, generator=g) * (0.1 if p.dim() == 1 else c**-0.5))
    z0 = torch.randn(1, n, n, c, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(1, n, generator=g) >= 0.1).to(DEV)

    def run(wait):
        z = z0
        with torch.no_grad():
            for i in range(6):
                if wait:
                    torch.cuda.synchronize()
                z = modules[i % 2](z * 0.5, mask)
        return z

    want = run(True)
    if graph:
        recorded = torch.cuda.CUDAGraph()
        with torch.cuda.graph(recorded):
            got = run(False)
        recorded.replay()
    else:
        got = run(False)
    assert torch.isfinite(want).all() and torch.equal(got, want)
