"""The prologue and the epilogues read z (the epilogues also the packed weights) while the kernel before them finishes. What a
call is given may have been written by the launch right before the call: stacks of calls, each on the output of the one before,
against the same calls with the device idle in between. The sizes give a CTA no, one, two and more tiles."""

import pytest
import torch

import miniworld_b200 as mw
from miniworld_b200 import functional as F_

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


@pytest.mark.parametrize("kind,c,drop", [("outgoing", 128, False), ("incoming", 64, False), ("bidirectional", 128, False),
                                         ("outgoing", 128, True), ("bidirectional", 128, True)])
@pytest.mark.parametrize("n", [8, 56, 136])
def test_two_parameter_sets_on_one_workspace(kind, c, drop, n):
    """Calls back to back with nothing between them, every one with other weights, LayerNorms and biases than the one before and
    the same workspace: each packs its own constants where those of the call before were read."""
    g = torch.Generator().manual_seed(n)
    module = KINDS[kind](c)
    outgoing = {"outgoing": True, "incoming": False, "bidirectional": None}[kind]
    z = torch.randn(1, n, n, c, generator=g).to(torch.bfloat16).to(DEV)
    scale = (torch.rand(1, n, c, generator=g) + 0.5).to(torch.bfloat16).to(DEV) if drop else None
    sets = []
    for _ in range(2):
        p = {k: (torch.randn(v.shape, generator=g) * (0.3 if v.dim() == 1 else v.shape[-1] ** -0.5) + (v.dim() == 1)).to(DEV)
             for k, v in module.named_parameters()}
        b = {k: torch.randn(p[f"{k}.weight"].shape[0], generator=g).to(DEV) for k in ("to_left", "to_right_gate", "to_gate", "to_out")}
        sets.append((p, F_._Weights(p, b, torch.device(DEV), bidirectional=outgoing is None, d_pair=c)))
    ws = F_.aligned_empty(F_.workspace_bytes(1, n, outgoing, c), torch.device(DEV))

    def run(out, wait=False):
        for i, y in enumerate(out):
            p, w = sets[i % 2]
            F_.trimul_forward(z, p, outgoing=outgoing, workspace=ws, out=y, weights=w, drop_scale=scale)
            if wait:
                torch.cuda.synchronize()

    want, got, replayed = ([torch.zeros_like(z) for _ in range(count)] for count in (2, 40, 40))
    run(want, wait=True)
    assert not torch.equal(*want) and all(torch.isfinite(w).all() for w in want)
    run(got)
    graph = torch.cuda.CUDAGraph()  # (no host time between the launches)
    with torch.cuda.graph(graph):
        run(replayed)
    for _ in range(3):
        graph.replay()
    assert all(torch.equal(y, want[i % 2]) for out in (got, replayed) for i, y in enumerate(out))


def _filled(kind, seed):
    """A module whose parameters are all non-zero (the default output gate and projection are zeros, behind which nothing shows)."""
    g = torch.Generator().manual_seed(seed)
    m = mw.Transition(128) if kind == "transition" else KINDS[kind](128)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_((1.0 if p.dim() == 1 else 0.0) + torch.randn(p.shape, generator=g) * (0.1 if p.dim() == 1 else p.shape[-1] ** -0.5))
    return m.to(DEV)


@pytest.mark.parametrize("kind", [*KINDS, "transition"])
@pytest.mark.parametrize("n", [8, 136])
def test_every_argument_written_by_the_launch_before(kind, n):
    """test_arguments_written_by_the_launch_before where each argument shows in the result: one of them is changed before every call,
    and every call gives another result."""
    g = torch.Generator().manual_seed(5)
    m = _filled(kind, n).to(torch.bfloat16).eval()
    z = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    mask = torch.ones(1, n, dtype=torch.bool, device=DEV)
    mask[:, n // 3] = False
    args = (z,) if kind == "transition" else (z, mask)
    changed = [*args, *m.parameters()]
    start = [t.detach().clone() for t in changed]

    def run(wait):
        out = []
        with torch.no_grad():
            for t, s in zip(changed, start):
                t.copy_(s)
            for t in changed:
                t.logical_not_() if t.dtype == torch.bool else t.add_(0.25)
                if wait:
                    torch.cuda.synchronize()
                out.append(m(*args))
                if wait:
                    torch.cuda.synchronize()
                if t.dtype == torch.bool:
                    t.logical_not_()
        return out

    want, got = run(True), run(False)
    assert all(torch.isfinite(w).all() and not torch.equal(w, z) for w in want)
    assert all(not torch.equal(a, b) for i, a in enumerate(want) for b in want[:i])
    assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("kind", [*KINDS, "transition"])
@pytest.mark.parametrize("n", [8, 136, 200])
def test_training_steps_with_every_gradient(kind, n):
    """test_training_steps_in_a_row where no gradient is zero: other parameters, input and output gradient in each step."""
    g = torch.Generator().manual_seed(n)
    m = _filled(kind, n + 1).to(torch.bfloat16).train()
    start = [p.detach().clone() for p in m.parameters()]
    z0 = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    dy0 = torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(1, n, generator=g) >= 0.1).to(DEV)

    def run(wait):
        z, out = z0.clone().requires_grad_(), []
        pause = torch.cuda.synchronize if wait else lambda: None
        for i in range(4):
            with torch.no_grad():
                for p, s in zip(m.parameters(), start):
                    p.copy_(s * (1 + 0.125 * i))
                z.copy_(z0 * (1 - 0.25 * i))
            pause()
            y = m(z) if kind == "transition" else m(z, mask)
            pause()
            dy = dy0 * (0.5 + 0.25 * i)
            pause()
            out.append([y.detach(), *torch.autograd.grad(y, [z, *m.parameters()], dy)])
            pause()
        return out

    want, got = run(True), run(False)
    for i, step in enumerate(want):
        assert all(torch.isfinite(t).all() and bool((t != 0).any()) for t in step)
        assert all(not torch.equal(a, b) for before in want[:i] for a, b in zip(step, before))
    assert all(torch.equal(a, b) for x, y in zip(want, got) for a, b in zip(x, y))


@pytest.mark.parametrize("kind", [*KINDS, "transition"])
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("before", ["copy", "memset", "other stream", "both streams"])
def test_what_may_come_before_a_call(kind, graph, before):
    """A call's first launch may overlap the kernel before it; what comes before it may also be a copy, a memset or another stream's
    work, eager and captured."""
    n = 72
    g = torch.Generator().manual_seed(3)
    m = _filled(kind, 4).to(torch.bfloat16).eval()
    src = [torch.randn(1, n, n, 128, generator=g).to(torch.bfloat16).to(DEV) for _ in range(3)]
    src[1].zero_()
    heavy = torch.randn(2048, 2048, device=DEV)
    z = torch.empty_like(src[0])
    side = torch.cuda.Stream()

    def fill(t):
        t.zero_() if before == "memset" else t.copy_(src[0])

    def run(wait):
        main = torch.cuda.current_stream()
        z.fill_(5.0)
        pause = torch.cuda.synchronize if wait else lambda: None
        if "stream" in before:
            side.wait_stream(main)
            with torch.cuda.stream(side):
                h = heavy @ heavy @ heavy  # (so that z comes late)
                fill(z)
            if before == "both streams":
                _ = src[2] * 2.0
            pause()
            main.wait_stream(side)
            h.record_stream(main)
        else:
            fill(z)
        pause()
        with torch.no_grad():
            y = m(z)
        pause()
        return y

    want = run(True).clone()
    for _ in range(5):
        if graph:
            torch.cuda.synchronize()
            recorded = torch.cuda.CUDAGraph()
            with torch.cuda.graph(recorded):
                got = run(False)
            z.fill_(5.0)
            recorded.replay()
        else:
            got = run(False)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and not torch.equal(want, z)
