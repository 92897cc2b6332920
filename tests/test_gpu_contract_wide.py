"""The contraction's tiles of up to 512 columns: lengths just above their smallest, with a last tile of 128 to 512 columns, rows
that fill half a tile and row ranges, in the three operand forms, against fp32 products per channel plane."""

import pytest
import torch

from miniworld_b200 import functional as F_

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SCALE = 0.0625  # the stored result is t * 2^-4


def _check(got, want):
    got = got.float() / SCALE
    assert torch.isfinite(got).all()
    # fp16 rounding of the stored value (2^-11 relative), and fp32 sums of up to 1000 products in another order
    assert bool(((got - want).abs() <= want.abs() * 2**-10 + 2e-3).all())


def _operands(B, N, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(B, N, 128, N, generator=g, device=DEV).to(torch.float16) for _ in range(3)]


def _status():
    return torch.zeros(16, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("B,N", [(1, 392), (2, 408), (1, 584), (1, 640), (1, 776), (1, 904)])
def test_contractions(B, N):
    left, right, _ = _operands(B, N, N)
    lf, rf = left.float().transpose(1, 2), right.float().transpose(1, 2)  # [B, 128, rows, N]
    for outgoing in (True, False):
        tri, st = torch.full_like(left, float("nan")), _status()
        F_.contract(left, right, tri, st, B, N, 0, N, outgoing)
        F_.check_status(st, "contract")
        _check(tri, (lf @ rf.mT if outgoing else lf.mT @ rf).transpose(1, 2))


@pytest.mark.parametrize("N", [392, 776])
@pytest.mark.parametrize("outgoing", [True, False])
def test_gradients_of_contractions(N, outgoing):
    left, right, dt = _operands(1, N, N + 1)
    dl, dr, st = torch.full_like(left, float("nan")), torch.full_like(left, float("nan")), _status()
    F_.contract_backward(dt, left, right, dl, dr, st, 1, N, outgoing)
    F_.check_status(st, "contract_backward")
    lf, rf, df = (t.float().transpose(1, 2) for t in (left, right, dt))
    _check(dl, (df @ rf if outgoing else rf @ df.mT).transpose(1, 2))
    _check(dr, (df.mT @ lf if outgoing else lf @ df).transpose(1, 2))


@pytest.mark.parametrize("outgoing", [True, False])
@pytest.mark.parametrize("begin,rows", [(0, 392), (8, 400), (104, 536)])
def test_row_ranges(begin, rows, outgoing):
    N = 640
    left, right, _ = _operands(1, N, begin + rows)
    lf, rf = left.float().transpose(1, 2), right.float().transpose(1, 2)
    want = (lf @ rf.mT if outgoing else lf.mT @ rf).transpose(1, 2)[:, begin : begin + rows]
    a = left[:, begin : begin + rows].contiguous() if outgoing else left  # (outgoing: the rows of the call only)
    tri, st = torch.full((1, rows, 128, N), float("nan"), dtype=torch.float16, device=DEV), _status()
    F_.contract(a, right, tri, st, 1, N, begin, rows, outgoing)
    F_.check_status(st, "contract")
    _check(tri, want)


@pytest.mark.parametrize("N", [1400, 1544])
def test_three_tiles_and_a_last_one_of_128_columns(N):
    """N = 1400 has tiles of 512, 512 and 384 columns, N = 1544 of 512, 512, 512 and 128 (a single part of 128): all three operand
    forms. (The tolerance holds there too: 97 accumulations of 16 products each, each off by 2^-23 of a sum of standard deviation 39
    at most a few times over, are 2e-3.)"""
    assert F_.contract_kernel(N, True) == F_.contract_kernel(N, False) == "contract_wide_kernel"
    left, right, dt = _operands(1, N, N)
    views = [t.transpose(1, 2) for t in (left, right, dt)]  # [1, 128, rows, N]

    def compare(got, form):
        for c in range(0, 128, 16):  # (in groups of channels: the fp32 copies of whole tensors are 1.2 GB each)
            _check(got.transpose(1, 2)[:, c : c + 16], form(*(v[:, c : c + 16].float() for v in views)))

    for outgoing in (True, False):
        tri, st = torch.full_like(left, float("nan")), _status()
        F_.contract(left, right, tri, st, 1, N, 0, N, outgoing)
        dl, dr = torch.full_like(left, float("nan")), torch.full_like(left, float("nan"))
        F_.contract_backward(dt, left, right, dl, dr, st, 1, N, outgoing)
        F_.check_status(st, "contract")
        if outgoing:
            compare(tri, lambda l, r, d: l @ r.mT)
            compare(dl, lambda l, r, d: d @ r)
            compare(dr, lambda l, r, d: d.mT @ l)
        else:
            compare(tri, lambda l, r, d: l.mT @ r)
            compare(dl, lambda l, r, d: r @ d.mT)
            compare(dr, lambda l, r, d: l @ d)


@pytest.mark.parametrize("B,N", [(1, 392), (2, 520), (1, 1032)])
def test_64_channels_of_a_row_of_128(B, N):
    """The narrow bidirectional module contracts channels 0-63 one way and 64-127 the other, in one set of planes."""
    g = torch.Generator().manual_seed(N)
    p = {f"to_{k}.weight": (torch.randn(128, 64, generator=g) * 0.3).to(DEV) for k in ("left", "left_gate", "right", "right_gate")}
    p["to_gate.weight"], p["to_out.weight"] = (torch.randn(64, k, generator=g).to(DEV) * k**-0.5 for k in (64, 128))
    for k, n in (("ln_pair", 64), ("ln_out", 128)):
        p[f"{k}.weight"], p[f"{k}.bias"] = torch.ones(n, device=DEV), torch.zeros(n, device=DEV)
    z = torch.randn(B, N, N, 64, generator=g).to(torch.bfloat16).to(DEV)
    ws = F_.aligned_empty(F_.workspace_bytes(B, N, None, 64), torch.device(DEV))
    F_.trimul_forward(z, p, None, outgoing=None, workspace=ws, check=True)
    off, count = F_.workspace_layout(B, N), B * N * 128 * N
    left, right, tri = (ws[o : o + count * 2].view(torch.float16).view(B, N, 128, N).transpose(1, 2).float() for o in off[2:])
    want = torch.cat([left[:, :64] @ right[:, :64].mT, left[:, 64:].mT @ right[:, 64:]], 1)
    assert bool((want != 0).any())
    _check(tri, want)
