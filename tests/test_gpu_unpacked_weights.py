"""A whole forward takes the weights of its first stage from the parameters and packs those of its last one on the way; the stages
called one by one read the packed block of a launch of its own. Both must give the same bits, in both weight types, with and
without biases, for grids of one pair of CTAs and more."""

import pytest
import torch

from miniworld_b200 import functional as F_

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _params(dtype, wide, seed, offset=0):
    g = torch.Generator().manual_seed(seed)

    def weight(*shape):
        w = (torch.randn(*shape, generator=g) * shape[1] ** -0.5).to(dtype)
        flat = torch.empty(w.numel() + offset, dtype=dtype, device=DEV)[offset:]
        return flat.view(shape).copy_(w)

    p = {f"to_{k}.weight": weight(wide, 128) for k in ("left", "left_gate", "right", "right_gate")}
    p["to_gate.weight"], p["to_out.weight"] = weight(128, 128), weight(128, wide)
    for k, n in (("ln_pair", 128), ("ln_out", wide)):
        p[f"{k}.weight"] = (1.0 + 0.1 * torch.randn(n, generator=g)).to(DEV)
        p[f"{k}.bias"] = (0.1 * torch.randn(n, generator=g)).to(DEV)
    biases = {k: 0.3 * torch.randn(wide if k in ("to_left", "to_left_gate", "to_right", "to_right_gate") else 128, generator=g).to(DEV)
              for k in ("to_left", "to_left_gate", "to_right_gate", "to_gate", "to_out")}
    return p, biases


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("biased", [False, True])
@pytest.mark.parametrize("bidir", [False, True])
@pytest.mark.parametrize("B,n", [(1, 8), (1, 72), (2, 136)])
def test_same_bits_as_the_stages(dtype, biased, bidir, B, n):
    p, biases = _params(dtype, 256 if bidir else 128, n)
    p["to_left.weight"].view(-1)[5] = float("inf")  # (clamped to the largest fp16 value)
    biases = biases if biased else None
    g = torch.Generator().manual_seed(1)
    z = torch.randn(B, n, n, 128, generator=g).to(torch.bfloat16).to(DEV)
    mask = (torch.rand(B, n, generator=g) >= 0.2).to(DEV)
    got = F_.trimul_forward(z, p, mask, outgoing=None if bidir else True, biases=biases, check=True)
    status = torch.zeros(16, dtype=torch.int32, device=DEV)
    left, right, t0, t1 = (torch.empty(B, n, 128, n, dtype=torch.float16, device=DEV) for _ in range(4))
    packed, packed_in = (F_.aligned_empty(F_.packed_bytes(), torch.device(DEV)) for _ in range(2))
    want = torch.empty_like(z)
    if bidir:
        F_.pack_weights_bidir(p, packed, packed_in, biases)
        F_.prologue(z, packed, left, right, status, token_mask=mask, has_bias=biased)
        F_.contract(left, right, t0, status, B, n, 0, n, True)
        F_.prologue(z, packed_in, left, right, status, token_mask=mask, has_bias=biased)
        F_.contract(left, right, t1, status, B, n, 0, n, False)
        F_.epilogue_wide(t0, t1, z, packed, packed_in, want, status)
    else:
        F_.pack_weights(p, packed, biases)
        F_.prologue(z, packed, left, right, status, token_mask=mask, has_bias=biased)
        F_.contract(left, right, t0, status, B, n, 0, n, True)
        F_.epilogue(t0, z, packed, want, status)
    F_.check_status(status, "stages")
    assert torch.isfinite(want).all() and torch.equal(got, want)


def test_backward_takes_weights_aligned_to_8_bytes():
    """(the bidirectional backward runs the first stage again; bf16 weights there need 8-byte alignment only)"""
    n = 24
    p, _ = _params(torch.bfloat16, 256, 3)
    q, _ = _params(torch.bfloat16, 256, 3, offset=4)
    z = torch.randn(1, n, n, 128, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV)
    ws = F_.aligned_empty(F_.workspace_bytes(1, n, None), torch.device(DEV))
    F_.trimul_forward(z, p, None, outgoing=None, workspace=ws)
    (dz0, g0), (dz1, g1) = (F_.trimul_backward(z, z, w, ws, None, outgoing=None, check=True) for w in (p, q))
    assert torch.equal(dz0, dz1) and all(torch.equal(g0[k], g1[k]) for k in g0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("biased", [False, True])
@pytest.mark.parametrize("bidir", [False, True])
@pytest.mark.parametrize("B,n", [(1, 8), (1, 80), (2, 136)])
def test_workspace_holds_the_packed_block(dtype, biased, bidir, B, n):
    """The second region of a forward's workspace is the block that a packing launch writes, whole: for a look at the stages it can
    be given to the first one."""
    p, biases = _params(dtype, 256 if bidir else 128, n)
    biases = biases if biased else None
    z = torch.randn(B, n, n, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    outgoing = None if bidir else False
    ws = F_.aligned_empty(F_.workspace_bytes(B, n, outgoing), torch.device(DEV)).fill_(0xA5)
    F_.trimul_forward(z, p, None, outgoing=outgoing, biases=biases, workspace=ws, check=True)
    want, other = (F_.aligned_empty(F_.packed_bytes(), torch.device(DEV)) for _ in range(2))
    F_.pack_weights_bidir(p, want, other, biases) if bidir else F_.pack_weights(p, want, biases)
    off = F_.workspace_layout(B, n)
    packed = ws[off[1] : off[1] + want.numel()]
    assert torch.equal(packed, want)
    if not bidir:  # (there the second half's planes are left behind)
        left, right = (torch.empty(B, n, 128, n, dtype=torch.float16, device=DEV) for _ in range(2))
        status = torch.zeros(16, dtype=torch.int32, device=DEV)
        F_.prologue(z, packed, left, right, status, has_bias=biased)
        F_.check_status(status, "prologue")
        for k, t in ((2, left), (3, right)):
            kept = ws[off[k] : off[k] + t.numel() * 2].view(torch.int16).view_as(t)
            assert torch.equal(kept, t.view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("outgoing", [True, None])
@pytest.mark.parametrize("n", [8, 80])
def test_workspace_holds_the_matrices_of_64_wide_pairs(dtype, outgoing, n):
    """(no packing entry point for these: the stored values are half the weights in fp16, the LayerNorm parameters as they are)"""
    g = torch.Generator().manual_seed(n)
    names = ("to_left", "to_left_gate", "to_right", "to_right_gate")
    p = {f"{k}.weight": (torch.randn(128, 64, generator=g) * 0.125).to(dtype).to(DEV) for k in names}
    p["to_gate.weight"], p["to_out.weight"] = ((torch.randn(64, k, generator=g) * k**-0.5).to(dtype).to(DEV) for k in (64, 128))
    for k, c in (("ln_pair", 64), ("ln_out", 128)):
        p[f"{k}.weight"], p[f"{k}.bias"] = torch.randn(c, generator=g).to(DEV), torch.randn(c, generator=g).to(DEV)
    z = torch.randn(1, n, n, 64, generator=g).to(torch.bfloat16).to(DEV)
    ws = F_.aligned_empty(F_.workspace_bytes(1, n, outgoing, 64), torch.device(DEV)).fill_(0xA5)
    F_.trimul_forward(z, p, None, outgoing=outgoing, workspace=ws, check=True)
    start = F_.workspace_layout(1, n)[1]
    got = ws[start : start + 4 * 128 * 64 * 2].view(torch.float16).view(4, 128, 64)
    assert torch.equal(got, torch.stack([(0.5 * p[f"{k}.weight"].float()).half() for k in names]))
    tail = ws[start + 6 * 32768 : start + F_.packed_bytes()].view(torch.float32)  # d [4][128], s / d of the epilogue, LayerNorm [2][128]
    assert bool((tail[:512] == 0).all())
    assert torch.equal(tail[1024 : 1024 + 64], p["ln_pair.weight"]) and torch.equal(tail[1152 : 1152 + 64], p["ln_pair.bias"])
