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


@pytest.mark.parametrize("kind", list(KINDS))
def test_arguments_written_by_the_launch_before(kind):
    """Parameters, masks and the pair tensor are changed in place right before every call."""
    g = torch.Generator().manual_seed(5)
    m = KINDS[kind](128).to(DEV).to(torch.bfloat16).eval()
    n = 136
    z = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(1, n, generator=g) >= 0.3).to(DEV)
    start = {k: v.detach().clone() for k, v in m.named_parameters()}
    z0, mask0 = z.clone(), mask.clone()

    def run(wait):
        out = []
        with torch.no_grad():
            for k, v in m.named_parameters():
                v.copy_(start[k])
            z.copy_(z0), mask.copy_(mask0)
            for i in range(8):
                changed = [z, mask, *m.parameters()]
                for t in changed[i % len(changed) :] + changed[: i % len(changed)]:  # each is the last one once
                    t.logical_not_() if t.dtype == torch.bool else t.mul_(-0.75)
                if wait:
                    torch.cuda.synchronize()
                out.append(m(z, mask))
                if wait:
                    torch.cuda.synchronize()
        return out

    assert all(torch.equal(a, b) for a, b in zip(run(True), run(False)))


@pytest.mark.parametrize("kind", [*KINDS, "transition"])
@pytest.mark.parametrize("n", [8, 136, 200])
def test_training_steps_in_a_row(kind, n):
    """The backward's kernels read what is older than the launch before them while that one finishes: steps without a pause, with
    z and the output's gradient written by the launches right before the passes, against steps with the device idle in between.
    (Every order of additions in a step is fixed.)"""
    g = torch.Generator().manual_seed(n)
    m = (mw.Transition(128) if kind == "transition" else KINDS[kind](128)).to(DEV).to(torch.bfloat16).train()
    z0 = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    dy0 = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(1, n, generator=g) >= 0.1).to(DEV)

    def run(wait):
        z, out = z0.clone().requires_grad_(), []
        pause = torch.cuda.synchronize if wait else lambda: None
        for i in range(4):
            with torch.no_grad():
                z.copy_(z0 * (1 - 0.25 * i))
            pause()
            y = m(z) if kind == "transition" else m(z, mask)
            pause()
            dy = dy0 * (0.5 + 0.25 * i)
            pause()
            out += torch.autograd.grad(y, [z, *m.parameters()], dy)
            pause()
        return out

    assert all(torch.equal(a, b) for a, b in zip(run(True), run(False)))
