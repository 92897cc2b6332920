"""Lengths that are not a multiple of 8 run without padding: the same bits as the same call on inputs padded with masked
tokens to the next multiple of 8 (which the functional entry points take), for outputs and input gradients."""

import pytest
import torch

import miniworld_b200 as mw
from miniworld_b200 import functional as F_
from miniworld_b200.training import trimul_train

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

KINDS = {
    "out": (lambda: mw.TriangleMultiplicationOutgoing(128), True),
    "in": (lambda: mw.TriangleMultiplicationIncoming(128), False),
    "bidir": (lambda: mw.BidirectionalTriangleMultiplication(128), None),
    "narrow_in": (lambda: mw.TriangleMultiplicationIncoming(64, 128), False),
    "narrow_bidir": (lambda: mw.BidirectionalTriangleMultiplication(64), None),
}


def _make(kind, B, N, seed):
    make, outgoing = KINDS[kind]
    g = torch.Generator().manual_seed(seed)
    m = make()
    for p in m.parameters():
        p.data = torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (p.dim() == 1) * 0.7
    m = m.to(DEV).train()
    z = torch.randn(B, N, N, m.d_pair, generator=g).to(torch.bfloat16).to(DEV)
    token = (torch.rand(B, N, generator=g) > 0.2).to(DEV)
    pair = (torch.rand(B, N, N, generator=g) > 0.2).to(DEV)
    return m, outgoing, z, token, pair


def _pad(t, dims, pad):
    return torch.nn.functional.pad(t, [0, 0] * (t.dim() - 1 - dims[-1]) + [0, pad] * len(dims))


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("B,N", [(1, 1), (1, 7), (2, 9), (2, 61), (1, 127), (1, 129), (1, 203), (1, 257), (1, 395)])
def test_ragged_equals_padded(kind, B, N):
    m, outgoing, z, token, pair = _make(kind, B, N, 900 + N)
    pad = (-N) % 8
    use_pair = kind in ("out", "in", "narrow_in") and N % 3 == 0
    zp = _pad(z, (1, 2), pad)
    tp, pp = _pad(token, (1,), pad), _pad(pair, (1, 2), pad)
    params = dict(m.named_parameters())
    dy = (torch.randn(z.shape, generator=torch.Generator().manual_seed(N)) * 0.02).to(torch.bfloat16).to(DEV)

    zr = z.clone().requires_grad_(True)
    y = m(zr, pair if use_pair else token)
    grads = torch.autograd.grad(y, [zr, *params.values()], dy)

    zq = zp.clone().requires_grad_(True)
    yq = trimul_train(zq, params, None if use_pair else tp, outgoing=outgoing, pair_mask=pp if use_pair else None)
    want = torch.autograd.grad(yq[:, :N, :N], [zq, *params.values()], dy)

    assert torch.equal(y, yq[:, :N, :N]) and y.is_contiguous()
    assert torch.equal(grads[0], want[0][:, :N, :N])
    for k, a, b in zip(params, grads[1:], want[1:]):
        # fp32 sums over the same terms, tile by tile in another order: 2^-24 times the square root of their number
        # (at most 395^2) is 2.4e-5 of the terms' size
        assert (a - b).norm() <= 1e-4 * b.norm().clamp_min(1e-6), k

    with torch.no_grad():  # the inference path, and no mask at all
        assert torch.equal(m.eval()(z, pair if use_pair else token), y)
        everything = torch.ones(B, N, dtype=torch.bool, device=DEV)
        assert torch.equal(m(z), m(z, everything))


def test_ragged_dropout_scale_and_no_residual():
    N = 45
    m, _, z, token, _ = _make("bidir", 2, N, 77)
    m.residual, m.p_drop = False, 0.25
    scale = ((torch.rand(2, 1, N, 128, generator=torch.Generator().manual_seed(1)) > 0.25).float() / 0.75).to(DEV)
    m._make_drop_row_scale = lambda pair, p: scale
    y = m(z, token)
    zp, tp = _pad(z, (1, 2), 3), _pad(token, (1,), 3)
    want = F_.trimul_forward(zp, dict(m.named_parameters()), tp, outgoing=None, residual=False,
                             drop_scale=torch.nn.functional.pad(scale, (0, 0, 0, 3)))
    assert torch.equal(y, want[:, :N, :N])
    with torch.no_grad():
        assert torch.equal(m(z, token), y)


def test_ragged_calls_take_what_they_took():
    """Storage that does not start on 16 bytes, masks that broadcast to the batch, inputs changed in place before the
    backward, output gradients that are slices: nothing of that is refused or changes the result at such a length."""
    N = 21
    m, _, z, token, _ = _make("out", 2, N, 78)
    with torch.no_grad():
        y = m(z, token)
        odd = torch.empty(z.numel() + 1, dtype=z.dtype, device=DEV)[1:].view(z.shape).copy_(z)
        assert odd.data_ptr() % 16 != 0 and torch.equal(m(odd, token), y)
        assert torch.equal(m(z, token[:1]), m(z, token[:1].expand(2, N)))
        assert torch.equal(m(z.transpose(1, 2), token), m(z.transpose(1, 2).contiguous(), token))
    dy = torch.randn(2, N, N, 128, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV) * 0.02
    want = torch.autograd.grad(m(zr := z.clone().requires_grad_(True), token), [zr], dy)[0]
    leaf = z.clone().requires_grad_(True)
    mid, mask = leaf * 1, token.clone()
    out = m(mid, mask)
    mid.data.mul_(2.0)
    mask.fill_(True)
    slab = torch.zeros(dy.numel() + 1, dtype=dy.dtype, device=DEV)[1:].view(dy.shape).copy_(dy)
    assert torch.equal(torch.autograd.grad(out, [leaf], slab)[0], want)
    with pytest.raises(RuntimeError):
        m(z, token[:, :-1])
    with pytest.raises(RuntimeError):  # the functional entry points keep their multiples of 8
        trimul_train(z, dict(m.named_parameters()), token)


def test_ragged_under_graph_capture():
    N = 43
    m, _, z, token, _ = _make("in", 1, N, 79)
    m = m.eval()
    with torch.no_grad():
        want = m(z, token)
        static = torch.zeros_like(z)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            m(static, token)
        torch.cuda.current_stream().wait_stream(s)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = m(static, token)
        static.copy_(z)
        g.replay()
        assert torch.equal(y, want)
