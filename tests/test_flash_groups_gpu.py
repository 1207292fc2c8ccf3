"""The two-group forward where its sequence of key tiles is short or uneven: items of a single key tile
(the groups take items in turn), of two and three, of all lengths under a causal mask, several items per CTA;
widths whose rows are stored 32 and 16 bytes at a time."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native
from test_flash_paths_gpu import BF, FP, test_flash_attention_paths as check

pytestmark = pytest.mark.gpu

# batch, sq, sk, heads, dim, dtype, how (c causal, k key padding, r relative table, g growing), dropout
CASES = [
    (2, 300, 100, 5, 64, BF, "", 0.1),
    (40, 200, 128, 8, 64, FP, "k", 0.0),
    (40, 129, 129, 8, 128, BF, "", 0.0),
    (30, 260, 384, 6, 64, BF, "g", 0.0),
    (2, 700, 700, 24, 32, BF, "c", 0.1),
    (3, 640, 640, 40, 64, FP, "cg", 0.0),
    (1, 1500, 260, 30, 128, FP, "c", 0.1),
    (2, 200, 300, 3, 40, FP, "c", 0.1),
    (2, 200, 300, 3, 72, BF, "", 0.0),
    (2, 140, 500, 3, 48, BF, "kr", 0.0),
]


@pytest.mark.parametrize("b,sq,sk,h,d,dtype,how,p", CASES)
def test_two_groups(b, sq, sk, h, d, dtype, how, p):
    check(b, sq, sk, h, d, dtype, how, p)


@pytest.mark.parametrize("d", [64, 128])
def test_scores_that_never_grow(d):
    """Equal scores: no row maximum grows after the first tile, so that nothing holds the accumulator's warps
    back but the product before.  The result is the mean of V: rounded once, as are P (exactly 1) and V."""
    b, s, h = 24, 640, 16
    q = torch.zeros(b, s, h, d, device="cuda", dtype=BF)
    v = torch.randn(b, s, h, d, device="cuda", dtype=BF)
    out = NF.flash_attention(q, q, v)
    assert native.ops().device_status() == 0
    want = v.double().mean(1, keepdim=True).expand(-1, s, -1, -1)
    err = (out.double() - want).abs()
    # bf16's half unit, and 32-bit sums of 640 terms
    assert (err <= want.abs() * 2.0 ** -8 + 640 * 2.0 ** -24 * v.abs().max()).all()
