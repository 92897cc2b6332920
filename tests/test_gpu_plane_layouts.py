"""Where a whole call's intermediates lie: the entry points of multiples of 8 and those of any length share a layout where both take
a length, also with each other's backward and with a workspace of just that size."""

import pytest
import torch

import miniworld_b200 as mw
from miniworld_b200 import functional as F_

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIRECTIONS = {"out": True, "in": False, "bidir": None}


def _setup(kind, n, c=128):
    g = torch.Generator().manual_seed(n)
    outgoing = DIRECTIONS[kind]
    m = mw.BidirectionalTriangleMultiplication(c, c) if outgoing is None else mw.TriangleMultiplication(c, 128, outgoing=outgoing)
    p = {k: ((1.0 if v.dim() == 1 else 0.0) + torch.randn(v.shape, generator=g) * (0.1 if v.dim() == 1 else v.shape[-1] ** -0.5)).to(DEV)
         for k, v in m.named_parameters()}
    z = torch.randn(2, n, n, c, generator=g).to(torch.bfloat16).to(DEV)
    dy = (torch.randn(z.shape, generator=g) * 0.01).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(2, n, generator=g) >= 0.1).to(DEV)
    return outgoing, p, z, dy, mask


def _forward(z, p, mask, outgoing, ws, any_n):
    return F_._forward(z, p, mask, outgoing, 1e-5, 1e-5, None, True, None, ws, None, True, None, None, any_n)


def _backward(dy, z, p, ws, mask, outgoing, any_n):
    return F_._backward(dy, z, p, ws, mask, outgoing, 1e-5, 1e-5, None, True, None, None, None, True, any_n)


@pytest.mark.parametrize("kind,c", [("out", 128), ("in", 64), ("bidir", 128), ("bidir", 64)])
@pytest.mark.parametrize("n", [8, 72, 136])
def test_forward_of_one_kind_and_backward_of_the_other(kind, c, n):
    outgoing, p, z, dy, mask = _setup(kind, n, c)
    results = []
    for forward_any in (False, True):
        for backward_any in (False, True):
            ws = F_.aligned_empty(F_._forward_need(2, n, outgoing, c), torch.device(DEV))
            y = _forward(z, p, mask, outgoing, ws, forward_any)
            dz, grads = _backward(dy, z, p, ws, mask, outgoing, backward_any)
            results.append([y, dz, *grads.values()])
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    assert all(torch.isfinite(t).all() and bool((t != 0).any()) for t in results[0])


@pytest.mark.parametrize("kind", ["out", "in"])
@pytest.mark.parametrize("n", [5, 43, 72, 130])
def test_stages_of_a_call_of_any_length(kind, n):
    """The layout of the length rounded up to a multiple of 8 finds left, right and tri of a call of any length."""
    outgoing, p, z, _, mask = _setup(kind, n)
    n8 = (n + 7) // 8 * 8
    ws = F_.aligned_empty(F_._forward_need(2, n8, outgoing, 128), torch.device(DEV))
    _forward(z, p, mask, outgoing, ws, True)
    off = F_.workspace_layout(2, n8)
    left, right, tri = (ws[o : o + 2 * n * 128 * n8 * 2].view(torch.float16).view(2, n, 128, n8)[..., :n].float() for o in off[2:])
    want = torch.einsum("bihk,bjhk->bihj" if outgoing else "bkhi,bkhj->bihj", left, right)
    # the stored result is t * 2^-4, rounded to fp16 once (2^-11 relative) from fp32 sums in another order
    assert bool(((tri / 0.0625 - want).abs() <= want.abs() * 2**-10 + 2e-3).all()) and bool((tri != 0).any())


@pytest.mark.parametrize("kind", list(DIRECTIONS))
@pytest.mark.parametrize("n", [8, 72, 200])
def test_workspaces_of_just_the_dense_size(kind, n):
    """The public calls take a workspace that ends with the dense planes (and refuse one byte less)."""
    outgoing, p, z, dy, mask = _setup(kind, n)
    off, plane = F_.workspace_layout(2, n), 2 * n * 128 * n * 2
    need = off[4] + plane + (plane + F_.packed_bytes() if outgoing is None else 0)
    assert need <= F_.workspace_bytes(2, n, outgoing)
    with pytest.raises(RuntimeError, match="workspace too small"):
        F_.trimul_forward(z, p, mask, outgoing=outgoing, workspace=F_.aligned_empty(need - 1, torch.device(DEV)))
    ws = F_.aligned_empty(need, torch.device(DEV))
    y = F_.trimul_forward(z, p, mask, outgoing=outgoing, workspace=ws, check=True)
    own = F_.aligned_empty(F_._backward_need(2, n, outgoing), torch.device(DEV))
    assert own.numel() <= F_.backward_workspace_bytes(2, n, outgoing)
    dz, _ = F_.trimul_backward(dy, z, p, ws, mask, outgoing=outgoing, workspace=own, check=True)
    assert torch.isfinite(y).all() and torch.isfinite(dz).all()


@pytest.mark.parametrize("n,general", [(40, "b200_trimul_forward_ex"), (43, "b200_trimul_forward_any")])
def test_an_error_names_the_entry_point_that_was_called(n, general):
    """(a weight whose storage starts off 16 bytes is refused by the C entry; a module that checks the status takes the general path)"""
    for check, name in ((False, "b200_trimul_forward_lines, for " + general), (True, general)):
        m = mw.TriangleMultiplication(128, 128, outgoing=True, check_status=check).to(DEV).to(torch.bfloat16).eval()
        w = m.to_gate.weight.detach()
        m.to_gate.weight.data = torch.empty(w.numel() + 1, dtype=w.dtype, device=DEV)[1:].view(w.shape).copy_(w)
        with torch.no_grad(), pytest.raises(RuntimeError, match="^" + name + ":"):
            m(torch.zeros(1, n, n, 128, dtype=torch.bfloat16, device=DEV), None)
