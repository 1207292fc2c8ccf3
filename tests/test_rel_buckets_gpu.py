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


@pytest.mark.parametrize("bidirectional", [True, False])
@pytest.mark.parametrize("buckets", list(range(6, 90, 3)) + [160, 200, 256])
def test_distances_on_borders(buckets, bidirectional):
    """Largest distances that are a square, cube or other power of a ratio times the exact buckets: distances
    fall on borders between buckets, where the last bit of the logarithm decides."""
    exact = buckets // (4 if bidirectional else 2)
    table = torch.zeros(buckets, 2, device="cuda")
    for far in sorted({exact * r ** e for r in (2, 3, 5, 6, 7, 10) for e in (1, 2, 3, 4)}
                      | {exact * a * a // 4 for a in range(3, 16)} | set(range(exact + 1, exact + 40))):
        if exact < far < 20000:
            got = native.ops().rel_buckets(table, 1500, 1500, bidirectional, 1.0 / exact,
                                           1.0 / math.log(far / exact))
            assert torch.equal(got, _distance_buckets("cuda", 1500, 1500, buckets, bidirectional, far)), far
