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
