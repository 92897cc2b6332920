"""The rule that picks the contraction's kernel, at the edges of its ranges."""

import pytest

from miniworld_b200 import functional as F_

PAIR, WIDE, ONE = "contract_pair_kernel", "contract_wide_kernel", "contract_kernel"


@pytest.mark.parametrize(
    "n,outgoing,incoming",
    [(64, ONE, ONE), (256, PAIR, PAIR), (384, ONE, ONE), (392, WIDE, WIDE), (448, PAIR, PAIR), (512, PAIR, PAIR), (640, WIDE, WIDE),
     (768, PAIR, PAIR), (896, WIDE, WIDE), (897, PAIR, WIDE), (1024, PAIR, WIDE), (1280, PAIR, PAIR), (1408, WIDE, WIDE),
     (1409, PAIR, WIDE), (1536, PAIR, WIDE), (1537, WIDE, WIDE), (1792, PAIR, PAIR), (2048, PAIR, WIDE), (2049, WIDE, WIDE)],
)
def test_kernel_of_a_length(n, outgoing, incoming):
    assert (F_.contract_kernel(n, True), F_.contract_kernel(n, False)) == (outgoing, incoming)
