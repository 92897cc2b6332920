"""One module called on several streams and from several threads at once: every call gives what it gives alone, and what a graph
captured keeps its memory."""

import threading

import pytest
import torch

import miniworld_b200 as mw

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

MAKE = {
    "out": lambda **k: mw.TriangleMultiplication(128, outgoing=True, **k),
    "bidir": lambda **k: mw.BidirectionalTriangleMultiplication(128, **k),
    "narrow": lambda **k: mw.TriangleMultiplication(64, 128, **k),
    "transition": lambda **k: mw.Transition(128, **k),
}


def _module(kind, N, count, **kw):
    g = torch.Generator().manual_seed(N)
    m = MAKE[kind](**kw)
    for p in m.parameters():
        p.data = torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (p.dim() == 1) * 0.7
    m = m.to(DEV).to(torch.bfloat16).eval()
    c = 64 if kind == "narrow" else 128
    inputs = [torch.randn(1, N, N, c, generator=g).to(torch.bfloat16).to(DEV) for _ in range(count)]
    with torch.no_grad():
        want = [m(z) for z in inputs]
    torch.cuda.synchronize()
    return m, inputs, want


@pytest.mark.parametrize("general", [False, True])  # True: the Python path (check_status selects it)
@pytest.mark.parametrize("kind", list(MAKE))
def test_two_streams(kind, general):
    m, inputs, want = _module(kind, 136, 2, check_status=general)
    streams = [torch.cuda.Stream() for _ in inputs]
    out = [[], []]
    with torch.no_grad():
        for _ in range(30):
            for z, s, o in zip(inputs, streams, out):
                with torch.cuda.stream(s):
                    o.append(m(z))
    torch.cuda.synchronize()
    for o, w in zip(out, want):
        assert all(torch.equal(y, w) for y in o)


@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("kind", list(MAKE))
def test_threads(kind, own_stream):
    m, inputs, want = _module(kind, 72, 4)
    out, errors = [[] for _ in inputs], []

    def work(i):
        try:
            stream = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
            with torch.no_grad(), torch.cuda.stream(stream):
                for _ in range(100):
                    out[i].append(m(inputs[i]))
        except Exception as e:  # (a failed assertion of the module would be lost with its thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(inputs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for o, w in zip(out, want):
        assert len(o) == 100 and all(torch.equal(y, w) for y in o)


@pytest.mark.parametrize("kind", list(MAKE))
def test_a_captured_call_keeps_its_memory(kind):
    """Warm-up and capture on one stream, then eager calls there and elsewhere, then other allocations: the graph's own scratch
    memory is not handed out."""
    m, inputs, want = _module(kind, 72, 2)
    z, static = inputs[0], torch.zeros_like(inputs[0])
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad():
        with torch.cuda.stream(s):
            m(static)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            y = m(static)
        assert m.device_status() == 0
        for stream in (s, torch.cuda.current_stream()):
            with torch.cuda.stream(stream):
                assert torch.equal(m(inputs[1]), want[1])
            torch.cuda.synchronize()
        filled = [torch.full((1 << 22,), 255, dtype=torch.uint8, device=DEV) for _ in range(64)]
        static.copy_(z)
        graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(y, want[0])
    assert all(bool((f == 255).all()) for f in filled)
