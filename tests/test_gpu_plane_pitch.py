"""Calls of the modules and of ``trimul_train`` keep their intermediates with rows of whole 128-byte lines, the functional entry
points keep dense ones: the results must not differ, at lengths on and off the lines and the tiles' edges."""

import pytest
import torch

import miniworld_b200 as mw
from miniworld_b200 import functional as F_
from miniworld_b200.training import trimul_train

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KINDS = {"out": (True, 128), "in": (False, 128), "bidir": (None, 128), "narrow_in": (False, 64), "narrow_bidir": (None, 64)}


def _module(kind):
    outgoing, c = KINDS[kind]
    if outgoing is None:
        return mw.BidirectionalTriangleMultiplication(c, 128 if c == 128 else 64)
    return mw.TriangleMultiplication(c, 128, outgoing=outgoing)


def _setup(kind, B, n):
    g = torch.Generator().manual_seed(n)
    m = _module(kind)
    c = KINDS[kind][1]
    with torch.no_grad():
        for p in m.parameters():
            p.copy_((1.0 if p.dim() == 1 else 0.0) + torch.randn(p.shape, generator=g) * (0.1 if p.dim() == 1 else c**-0.5))
    z = torch.randn(B, n, n, c, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(B, n, generator=g) >= 0.1).to(DEV)
    dy = (torch.randn(z.shape, generator=g) * 0.01).to(torch.bfloat16).to(DEV)
    return m.to(DEV), z, mask, dy


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("B,n", [(1, 8), (2, 56), (1, 64), (1, 72), (2, 120), (1, 136), (1, 200), (1, 264)])
def test_padded_rows_change_nothing(kind, B, n):
    m, z, mask, dy = _setup(kind, B, n)
    params = dict(m.named_parameters())
    with torch.no_grad():
        got = m.eval()(z, mask)
        want = F_.trimul_forward(z, {k: v.detach() for k, v in params.items()}, mask, outgoing=KINDS[kind][0])
    assert torch.equal(got, want)
    zr = z.clone().requires_grad_(True)
    steps = []
    for check in (False, True):  # a call that checks the status takes the general path, whose workspace is dense
        y = trimul_train(zr, params, mask, outgoing=KINDS[kind][0], check=check)
        steps.append(torch.autograd.grad(y, [zr, *params.values()], dy))
    for a, b in zip(*steps):
        assert torch.equal(a, b)


def test_workspace_sizes():
    for n in (8, 64, 72, 200, 256):
        dense, rows = F_.workspace_layout(2, n), 2 * n * 128 * 2
        pitch = (n + 63) // 64 * 64
        assert F_.workspace_bytes(2, n) == dense[2] + 3 * rows * pitch  # enough for either kind of call
        with pytest.raises(RuntimeError, match="workspace too small"):
            m, z, mask, _ = _setup("out", 2, n)
            F_.trimul_forward(z, dict(m.named_parameters()), mask, workspace=torch.empty(dense[4], dtype=torch.uint8, device=DEV))
