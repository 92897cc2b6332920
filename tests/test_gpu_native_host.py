"""The native host path of the modules against the general Python path (which ``check_status`` selects): the same kernels on
the same arguments, so the same bits; and calls the native path leaves to the general one. Which path a call took is counted at
the native entry points."""

import pytest
import torch
from torch import nn

import miniworld_b200 as mw
from miniworld_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

MAKE = {
    "out": lambda **k: mw.TriangleMultiplication(128, outgoing=True, **k),
    "in": lambda **k: mw.TriangleMultiplicationIncoming(128, **k),
    "bidir": lambda **k: mw.BidirectionalTriangleMultiplication(128, **k),
    "narrow": lambda **k: mw.TriangleMultiplication(64, 128, **k),
    "narrow_bidir": lambda **k: mw.BidirectionalTriangleMultiplication(64, **k),
    "transition": lambda **k: mw.Transition(128, **k),
}


def _pair(kind, dtype, **kw):
    """The same module twice: native host path, general path."""
    g = torch.Generator().manual_seed(len(kind))
    a, b = MAKE[kind](**kw), MAKE[kind](check_status=True, **kw)
    for p in a.parameters():
        p.data = torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (p.dim() == 1) * 0.7
    b.load_state_dict(a.state_dict())
    return a.to(DEV).to(dtype), b.to(DEV).to(dtype)


def _input(kind, B=2, N=40, seed=5):
    g = torch.Generator().manual_seed(seed)
    c = 64 if kind.startswith("narrow") else 128
    z = torch.randn(B, N, N, c, generator=g).to(torch.bfloat16).to(DEV)
    return z, (torch.rand(B, N, generator=g) > 0.2).to(DEV), (torch.randn(z.shape, generator=g) * 0.02).to(torch.bfloat16).to(DEV)


class _Counted:
    """The native module; ``taken`` and ``left`` count the calls it served and the ones it answered with None."""

    def __init__(self, module):
        self.module, self.taken, self.left = module, 0, 0

    def __getattr__(self, name):
        f = getattr(self.module, name)

        def call(*args):
            out = f(*args)
            if out is None:
                self.left += 1
            else:
                self.taken += 1
            return out

        return call

    def __call__(self, f):
        """(calls served, calls left) by the native module while ``f`` runs."""
        before = self.taken, self.left
        f()
        return self.taken - before[0], self.left - before[1]


@pytest.fixture
def native(monkeypatch):
    counted = _Counted(_lib.native())
    monkeypatch.setattr(_lib, "_native", counted)
    return counted


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N", [40, 43])
@pytest.mark.parametrize("kind", list(MAKE))
def test_same_bits_as_the_general_path(kind, N, dtype, native):
    a, b = _pair(kind, dtype)
    z, mask, dy = _input(kind, N=N)
    args = () if kind == "transition" else (mask,)
    with torch.no_grad():
        assert torch.equal(a.eval()(z, *args), b.eval()(z, *args))
        assert (native.taken, native.left) == (1, 0)  # a's call; b did not ask
    grads = []
    for m in (a.train(), b.train()):
        zr = z.clone().requires_grad_(True)
        y = m(zr, *args)
        grads.append([y.detach(), *torch.autograd.grad(y, [zr, *m.parameters()], dy)])
    assert (native.taken, native.left) == (2, 0)
    for x, y in zip(*grads):
        assert x.dtype == y.dtype and torch.equal(x, y)


def test_calls_left_to_the_general_path(native):
    a, b = _pair("in", torch.bfloat16)
    z, mask, _ = _input("in")
    with torch.no_grad():
        want = b.eval()(z, mask)
        a = a.eval()
        assert native(lambda: a(z, mask)) == (1, 0)
        for m in (mask.to(torch.uint8), mask.float(), mask.cpu()):
            assert native(lambda: a(z, m)) == (0, 1)
            assert torch.equal(a(z, m), want)
        assert torch.equal(a(z.float(), mask), want.float()) and native(lambda: a(z.float(), mask)) == (0, 1)
        zt = z.transpose(1, 2).contiguous().transpose(1, 2)
        assert not zt.is_contiguous() and torch.equal(a(zt, mask), want) and native(lambda: a(zt, mask)) == (0, 1)
        pair = (mask[:, :, None] & mask[:, None, :])
        assert torch.equal(a(z, pair), want) and torch.equal(a(z, pair.transpose(1, 2)), want)
        taken = native.taken
        for bad in (z[:, :-1], z.cpu(), z[..., :64], z[0]):
            with pytest.raises(RuntimeError):
                a(bad, mask)
        with pytest.raises(RuntimeError):
            a(z, mask[:, :-1])
        a.to_left.weight.data = a.to_left.weight.data.t().contiguous().t()
        with pytest.raises(RuntimeError):
            a(z, mask)
        assert native.taken == taken


@pytest.mark.parametrize("N,entry", [(40, "b200_trimul_forward_ex"), (43, "b200_trimul_forward_any")])
def test_an_error_names_the_entry_point(N, entry):
    """(a weight whose storage starts off 16 bytes is refused by the C entry, on either path)"""
    for m in _pair("out", torch.float32):
        w = m.to_gate.weight.detach()
        m.to_gate.weight.data = torch.empty(w.numel() + 1, device=DEV)[1:].view(w.shape).copy_(w)
        with torch.no_grad(), pytest.raises(RuntimeError, match=entry + ":"):
            m.eval()(_input("out", N=N)[0])


def test_reparametrised_and_swapped_parameters(native):
    a, b = _pair("out", torch.float32)
    z, mask, _ = _input("out")

    class Twice(nn.Module):
        def forward(self, w):
            return 2.0 * w

    torch.nn.utils.parametrize.register_parametrization(a.to_left, "weight", Twice())
    b.to_left.weight.data.mul_(2.0)
    with torch.no_grad():
        assert torch.equal(a.eval()(z, mask), b.eval()(z, mask))
        assert native.taken == 0
    c, d = _pair("out", torch.float32)
    new = {"to_gate.weight": torch.randn(128, 128, device=DEV) * 0.1}
    d.to_gate.weight.data.copy_(new["to_gate.weight"])
    with torch.no_grad():
        assert torch.equal(torch.func.functional_call(c.eval(), new, (z, mask)), d.eval()(z, mask))


def test_graph_behaviour(native):
    a, b = _pair("bidir", torch.float32, p_drop=0.25)
    z, mask, dy = _input("bidir")
    scale = ((torch.rand(2, 1, 40, 128, generator=torch.Generator().manual_seed(1)) > 0.25).float() / 0.75).to(torch.bfloat16).to(DEV)
    a._make_drop_row_scale = b._make_drop_row_scale = lambda pair, p: scale
    a, b = a.train(), b.train()
    # parameters only, a subset of the gradients, an expanded output gradient
    y = a(z, mask)
    assert (native.taken, native.left) == (1, 0) and "TriMulFunction" not in type(y.grad_fn).__name__
    got = torch.autograd.grad(y, [a.to_out.weight, a.ln_pair.bias], dy[:1].expand_as(dy))
    want = torch.autograd.grad(b(z, mask), [b.to_out.weight, b.ln_pair.bias], dy[:1].expand_as(dy).contiguous())
    assert all(torch.equal(p, q) for p, q in zip(got, want))
    # a second backward through the same forward is refused, with and without the graph kept
    for keep in (True, False):
        y = a(z, mask)
        y.backward(dy, retain_graph=keep)
        with pytest.raises(RuntimeError):
            y.backward(dy)
    # the saved tensors go through hooks; a parameter changed in place since the forward is noticed
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(DEV)):
        y = a(z, mask)
    assert len(packed) == 11
    hooked = torch.autograd.grad(y, [a.to_out.weight, a.ln_pair.bias], dy)
    want = torch.autograd.grad(b(z, mask), [b.to_out.weight, b.ln_pair.bias], dy)
    assert all(torch.equal(p, q) for p, q in zip(hooked, want))
    y = a(z, mask)
    with torch.no_grad():
        a.to_out.weight.mul_(1.5)
    with pytest.raises(RuntimeError):
        y.backward(dy)
    with torch.no_grad():
        assert not a(z, mask).requires_grad
    # another stream than the default one
    b.to_out.weight.data.copy_(a.to_out.weight.data)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        zr = z.clone().requires_grad_(True)
        g = torch.autograd.grad(a(zr, mask), zr, dy)[0]
    torch.cuda.current_stream().wait_stream(s)
    zr = z.clone().requires_grad_(True)
    assert torch.equal(g, torch.autograd.grad(b(zr, mask), zr, dy)[0])


@pytest.mark.parametrize("kind", ["triangle", "transition"])
@pytest.mark.parametrize("train", [False, True])
def test_dispatch_modes_see_the_allocations(kind, train):
    """Under a mode whose tensors have no memory a call is refused and nothing runs; a mode that only looks on changes nothing."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        empties = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.empties += "empty" in str(func)
            return func(*args, **(kwargs or {}))

    m = mw.Transition(128) if kind == "transition" else mw.TriangleMultiplication(128, 128, outgoing=True)
    m = m.to(DEV).to(torch.bfloat16).train(train)
    z = torch.randn(1, 40, 40, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    mask = torch.ones(1, 40, dtype=torch.bool, device=DEV)
    args = (z,) if kind == "transition" else (z, mask)
    with torch.set_grad_enabled(train):
        want = m(*args)
        with Count() as count:
            got = m(*args)
        assert torch.equal(got, want) and count.empties > 0
        with FakeTensorMode(allow_non_fake_inputs=True), pytest.raises(RuntimeError):
            m(*args)
        assert torch.equal(m(*args), want)
