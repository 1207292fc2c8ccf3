"""T5's distance buckets from the kernel: the numbers that the operators give, at every distance."""
import math

import pytest
import torch

from slapo_b200.ops import native
from slapo_b200.ops.flash_attn import _distance_buckets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bidirectional", [True, False])
@pytest.mark.parametrize("buckets", [4, 5, 7, 8, 16, 32, 33, 48, 64, 128])
@pytest.mark.parametrize("max_distance", [16, 20, 64, 128, 129, 256, 1000])
def test_buckets(buckets, max_distance, bidirectional):
    exact = buckets // (4 if bidirectional else 2)
    if max_distance <= exact:
        pytest.skip("torch's to report")
    table = torch.zeros(buckets, 2, device="cuda")
    for sq, sk in ((1, 1), (1, 1500), (700, 1), (300, 2100), (1100, 1100)):
        got = native.ops().rel_buckets(table, sq, sk, bidirectional, 1.0 / exact,
                                       1.0 / math.log(max_distance / exact))
        want = _distance_buckets("cuda", sq, sk, buckets, bidirectional, max_distance)
        assert torch.equal(got, want), (sq, sk)
