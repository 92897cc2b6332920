"""Backward kernels where their tilings and reductions have edges: position counts around one tile and around one tile per
CTA for the Transition, short rows for the wide LayerNorm statistics, and gradients of zero or with a non-finite value for the
scale, against float64 torch on the GPU.

Bound: an input gradient is rounded to bf16 (relative 2^-9 / sqrt(3) = 1.1e-3, up to 1.7e-3 by how values lie in their
binades) after three fp16 roundings (2^-12 each, through products): 2.5 times their sum."""

import pytest
import torch
import torch.nn.functional as F

import miniworld_b200 as mw

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 5e-3


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


def _transition64(m, x, dy):
    p = {k: v.detach().double().requires_grad_(True) for k, v in m.named_parameters()}
    z = x.double().requires_grad_(True)
    h = F.layer_norm(z, (128,), p["ln_in.weight"], p["ln_in.bias"], 1e-5)
    y = z + F.linear(F.silu(F.linear(h, p["expand_a.weight"])) * F.linear(h, p["expand_b.weight"]), p["squeeze.weight"])
    return torch.autograd.grad(y, [z, *p.values()], dy.double())


def _module(make, seed):
    g = torch.Generator().manual_seed(seed)
    m = make()
    for p in m.parameters():
        p.data = torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (p.dim() == 1) * 0.7
    return m.to(DEV).train(), g


@pytest.mark.parametrize("positions", [1, 127, 128, 129, 147 * 128 + 1, 148 * 128, 148 * 128 + 1, 4 * 148 * 128 + 77])
def test_transition_position_counts(positions):
    m, g = _module(lambda: mw.Transition(128), positions)
    x = torch.randn(positions, 128, generator=g).to(torch.bfloat16).to(DEV)
    dy = (torch.randn(positions, 128, generator=g) * 0.02).to(torch.bfloat16).to(DEV)
    xr = x.clone().requires_grad_(True)
    got = torch.autograd.grad(m(xr), [xr, *m.parameters()], dy)
    for name, a, b in zip(["x", *dict(m.named_parameters())], got, _transition64(m, x, dy)):
        assert _rel(a, b) <= TOL, (name, _rel(a, b))


@pytest.mark.parametrize("positions", [128, 148 * 128, 2 * 148 * 128])
def test_transition_last_tile_repeats(positions):
    """The first launch stores x_hat of a block's last tile (of its only one at up to 148 tiles) for the three launches after it
    while the block gathers its column sums: the copy must not see them, in any of forty calls."""
    m, g = _module(lambda: mw.Transition(128), positions)
    x = torch.randn(positions, 128, generator=g).to(torch.bfloat16).to(DEV)
    dy = (torch.randn(positions, 128, generator=g) * 0.02).to(torch.bfloat16).to(DEV)

    def grads():
        xr = x.clone().requires_grad_(True)
        return torch.autograd.grad(m(xr), [xr, *m.parameters()], dy)

    first = grads()
    for a, b in zip(first, _transition64(m, x, dy)):
        assert _rel(a, b) <= TOL
    for _ in range(39):
        assert all(torch.equal(a, b) for a, b in zip(first, grads()))


def _triangle64(m, z, dy):
    """Gradients of the bidirectional module in float64."""
    p = {k: v.detach().double().requires_grad_(True) for k, v in m.named_parameters()}
    x = z.double().requires_grad_(True)
    h = F.layer_norm(x, (128,), p["ln_pair.weight"], p["ln_pair.bias"], 1e-5)
    left = torch.sigmoid(F.linear(h, p["to_left_gate.weight"])) * F.linear(h, p["to_left.weight"])
    right = torch.sigmoid(F.linear(h, p["to_right_gate.weight"])) * F.linear(h, p["to_right.weight"])
    t = torch.cat([torch.einsum("bikd,bjkd->bijd", left[..., :128], right[..., :128]),
                   torch.einsum("bkid,bkjd->bijd", left[..., 128:], right[..., 128:])], -1)
    t = F.layer_norm(t, (256,), p["ln_out.weight"], p["ln_out.bias"], 1e-5)
    y = x + torch.sigmoid(F.linear(h, p["to_gate.weight"])) * F.linear(t, p["to_out.weight"])
    return torch.autograd.grad(y, [x, *p.values()], dy.double())


@pytest.mark.parametrize("B,N", [(1, 8), (3, 8), (1, 24), (1, 136), (2, 40)])
def test_wide_statistics_of_short_rows(B, N):
    """The bidirectional module's gradients against float64 where its statistics kernel has edges (a block takes eight groups of
    eight columns, across rows and samples); and they do not depend on the batch they are computed in."""
    m, g = _module(lambda: mw.BidirectionalTriangleMultiplication(128), 7 * N)
    z = torch.randn(B, N, N, 128, generator=g).to(torch.bfloat16).to(DEV)
    dy = (torch.randn(B, N, N, 128, generator=g) * 0.02).to(torch.bfloat16).to(DEV)
    dy[..., 0, 0, 0] = 0.5  # the same largest value, hence the same scale, in every sample

    def grad(a, b):
        a = a.clone().requires_grad_(True)
        return torch.autograd.grad(m(a), a, b)[0]

    whole = grad(z, dy)
    assert _rel(whole, _triangle64(m, z, dy)[0]) <= TOL
    for i in range(B):
        assert torch.equal(whole[i : i + 1], grad(z[i : i + 1], dy[i : i + 1]))


@pytest.mark.parametrize("make,shape", [(lambda: mw.Transition(128), (300, 128)), (lambda: mw.TriangleMultiplication(128), (1, 24, 24, 128))])
def test_scale_of_special_gradients(make, shape):
    m, g = _module(make, 5)
    x = torch.randn(*shape, generator=g).to(torch.bfloat16).to(DEV).requires_grad_(True)
    dy = (torch.randn(*shape, generator=g) * 0.02).to(torch.bfloat16).to(DEV)
    for t in torch.autograd.grad(m(x), [x, *m.parameters()], torch.zeros_like(dy)):
        assert torch.equal(t, torch.zeros_like(t))
    # a power of two through the whole backward: exactly that power in every gradient
    a = torch.autograd.grad(m(x), [x, *m.parameters()], dy)
    b = torch.autograd.grad(m(x), [x, *m.parameters()], dy * 2.0**-20)
    for u, v in zip(a, b):
        assert torch.equal(u * 2.0**-20, v)
    # an infinity does not set the scale: the finite gradients stay finite where it does not reach
    bad = dy.clone()
    bad.view(-1, 128)[-1, 3] = float("inf")
    out = torch.autograd.grad(m(x), x, bad)[0]
    # the Transition works position by position; the triangle update (outgoing) passes a gradient at (i, j) on to row i through
    # left and to row j through right, which is the last row twice
    reached = -1 if len(shape) == 2 else (slice(None), -1)
    clean = torch.ones_like(out, dtype=torch.bool)
    clean[reached] = False
    assert torch.equal(out[clean], a[0][clean]) and bool(torch.isfinite(out[clean]).all())
