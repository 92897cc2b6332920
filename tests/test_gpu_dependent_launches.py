"""Launches overlap the kernel before them on the stream. A kernel that reads, through the SMs' L1, what that one has read there and
then overwritten must not be answered by the old lines: chains of calls in place against the same chains out of place."""

import pytest
import torch

from miniworld_b200 import functional as F_

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offset", [0, 8])  # elements: 32-byte and 16-byte aligned rows
@pytest.mark.parametrize("positions", [256, 148 * 128, 4 * 148 * 128 + 77])
def test_transition_chain_in_place(positions, offset):
    """Every call's input is the output of the launch before it (the weights are packed once), written over that one's input."""
    g = torch.Generator().manual_seed(positions)
    params = {"ln_in.weight": torch.ones(128), "ln_in.bias": torch.zeros(128), "expand_a.weight": torch.randn(512, 128, generator=g) / 11,
              "expand_b.weight": torch.randn(512, 128, generator=g) / 11, "squeeze.weight": torch.randn(128, 512, generator=g) / 22}
    packed = F_.aligned_empty(F_.transition_packed_bytes(), torch.device(DEV))
    status = torch.zeros(16, dtype=torch.int32, device=DEV)
    F_.transition_pack_weights({k: v.to(DEV) for k, v in params.items()}, packed)
    x = torch.randn(positions, 128, generator=g).to(torch.bfloat16).to(DEV)
    want = [x]
    for _ in range(20):
        want.append(F_.transition_forward(want[-1], packed, status))
        torch.cuda.synchronize()
    buf = torch.empty(positions * 128 + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(positions, 128).copy_(x)
    for _ in range(20):
        F_.transition_forward(buf, packed, status, out=buf)
    assert torch.equal(buf, want[-1])
    assert F_.read_status(status) == 0
