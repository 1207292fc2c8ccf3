"""Attention at the edges of the backward's half tiles (64 streamed rows that two groups of warps
take in turn): items of one half tile, of an odd number, and the diagonal on their borders."""
import pytest
import torch

from test_flash_paths_gpu import test_flash_attention_paths as _check

pytestmark = pytest.mark.gpu

# (T5's table is tested at the lengths of the other file: at 64 x 1100 most keys share the last bucket,
# whose gradient is what is left of near-equal sums - delta comes from outputs rounded to 16 bits, so
# that its error, 2^-9 |O| |dO| P(bucket) per row, has nothing to cancel against: 1.4e-2 for any kernel.)
LENGTHS = [(1, 65), (63, 64), (64, 63), (65, 65), (127, 193), (193, 127), (320, 320), (64, 700)]


@pytest.mark.parametrize("sq,sk", LENGTHS)
@pytest.mark.parametrize("d,how,p", [(64, "", 0.1), (64, "c", 0.0), (128, "c", 0.1), (128, "k", 0.0),
                                     (80, "ck", 0.1)])
def test_half_tiles(sq, sk, d, how, p):
    _check(2, sq, sk, 3, d, torch.bfloat16, how, p)


# more work items than CTAs, of one and of an odd number of half tiles: a group's turn moves from
# item to item
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("sq,sk", [(60, 60), (150, 150)])
def test_turns_over_items(sq, sk, d):
    _check(40, sq, sk, 8, d, torch.bfloat16, "", 0.1)
