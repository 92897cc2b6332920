"""Outputs and gradients of training steps against recorded digests: a change of the backward kernels' structure (which thread
does what, in which launch) must keep every rounding and every order of additions, so that a run can be repeated bit for bit
with a later build.

The digests in ``golden/backward_bits.json`` were taken on a B200 (148 SMs) from the build at commit a13228c, whose kernels had
another structure. Run as a program, this file prints the digests of the build that it finds. The sizes put the tile counts
below, at and above one tile per CTA, and the numbers of partial sums at and off multiples of 16 (the groups they are added in).
"""

import hashlib
import json
from pathlib import Path

import pytest
import torch

from miniworld_b200.training import transition_train, trimul_train

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GOLDEN = Path(__file__).resolve().parent / "golden" / "backward_bits.json"

# name: (direction or "transition", d_pair, B, N or positions, mask, dropout, parameters' type)
CASES = {
    "out_n8": (True, 128, 1, 8, None, False, torch.float32),
    "out_n104": (True, 128, 1, 104, "token", False, torch.float32),
    "out_n192": (True, 128, 1, 192, "token", True, torch.float32),
    "in_b2_n72": (False, 128, 2, 72, "pair", False, torch.float32),
    "in_n264_bf16": (False, 128, 1, 264, "pair", False, torch.bfloat16),
    "bidir_b2_n24": (None, 128, 2, 24, "token", False, torch.float32),
    "bidir_n136": (None, 128, 1, 136, None, False, torch.float32),
    "bidir_n160_drop": (None, 128, 1, 160, "token", True, torch.float32),
    "narrow_out_n136": (True, 64, 1, 136, "pair", False, torch.float32),
    "narrow_bidir_b2_n88": (None, 64, 2, 88, "token", False, torch.float32),
    "transition_1": ("transition", 128, 1, 1, None, False, torch.float32),
    "transition_300": ("transition", 128, 1, 300, None, False, torch.float32),
    "transition_14075": ("transition", 128, 1, 14075, None, False, torch.bfloat16),
    "transition_37965": ("transition", 128, 1, 37965, None, False, torch.float32),
    "transition_147456": ("transition", 128, 1, 147456, None, False, torch.float32),
}


def _step(name):
    op, c, b, n, mask, drop, dtype = CASES[name]
    g = torch.Generator().manual_seed(sum(map(ord, name)))

    def param(*shape):
        r = torch.randn(*shape, generator=g)
        return (1.0 + 0.1 * r if len(shape) == 1 else (r * shape[1] ** -0.5).to(dtype)).to(DEV).requires_grad_(True)

    if op == "transition":
        shape = (n, c)
        params = {"ln_in.weight": param(c), "ln_in.bias": param(c), "expand_a.weight": param(4 * c, c),
                  "expand_b.weight": param(4 * c, c), "squeeze.weight": param(c, 4 * c)}
    else:
        shape = (b, n, n, c)
        w = 256 if op is None and c == 128 else 128
        params = {"ln_pair.weight": param(c), "ln_pair.bias": param(c), "to_left.weight": param(w, c),
                  "to_left_gate.weight": param(w, c), "to_right.weight": param(w, c), "to_right_gate.weight": param(w, c),
                  "ln_out.weight": param(w), "ln_out.bias": param(w), "to_gate.weight": param(c, c), "to_out.weight": param(c, w)}
    z = (torch.randn(shape, generator=g) * (0.5 + 1.5 * torch.rand(c, generator=g))).to(torch.bfloat16).to(DEV).requires_grad_(True)
    dy = (torch.randn(shape, generator=g) * 0.01).to(torch.bfloat16).to(DEV)
    if op == "transition":
        y = transition_train(z, params)
    else:
        token = (torch.rand(b, n, generator=g) >= 0.1).to(DEV) if mask == "token" else None
        pair = (torch.rand(b, n, n, generator=g) >= 0.1).to(DEV) if mask == "pair" else None
        scale = ((torch.rand(b, 1, n, c, generator=g) >= 0.25).to(torch.bfloat16) / 0.75).to(DEV) if drop else None
        y = trimul_train(z, params, token, outgoing=op, pair_mask=pair, drop_scale=scale)
    return {"y": y.detach(), "z": None, **dict.fromkeys(params)}, torch.autograd.grad(y, [z, *params.values()], dy)


def digests(name):
    out, grads = _step(name)
    out.update(zip(list(out)[1:], grads))
    # (+ 0.0: both zeros alike)
    return {k: hashlib.sha256((v.float() + 0.0).cpu().numpy().tobytes()).hexdigest()[:16] for k, v in out.items()}


@pytest.mark.parametrize("name", list(CASES))
def test_same_bits(name):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the order of the partial sums depends on the number of SMs; recorded with 148")
    want, got = json.loads(GOLDEN.read_text())[name], digests(name)
    assert got == want, sorted(k for k in want if got[k] != want[k])


if __name__ == "__main__":
    print(json.dumps({name: digests(name) for name in CASES}, indent=1))
