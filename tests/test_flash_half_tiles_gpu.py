"""Attention at the edges of the backward's half tiles (64 streamed rows that two groups of warps
take in turn): items of one half tile, of an odd number, and the diagonal on their borders."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native
from test_flash_paths_gpu import TOL, _reference
from test_flash_paths_gpu import test_flash_attention_paths as _check

pytestmark = pytest.mark.gpu

LENGTHS = [(1, 65), (63, 64), (64, 63), (65, 65), (127, 193), (193, 127), (320, 320), (64, 700)]


@pytest.mark.parametrize("sq,sk", LENGTHS)
@pytest.mark.parametrize("d,how,p", [(64, "", 0.1), (64, "c", 0.0), (128, "c", 0.1), (128, "k", 0.0),
                                     (80, "ck", 0.1)])
def test_half_tiles(sq, sk, d, how, p):
    _check(2, sq, sk, 3, d, torch.bfloat16, how, p)


@pytest.mark.parametrize("sq,sk", LENGTHS[:-1])
def test_half_tiles_with_a_table(sq, sk):
    _check(2, sq, sk, 3, 64, torch.bfloat16, "ckr", 0.1)


@pytest.mark.parametrize("d,causal,sk", [(64, True, 700), (64, True, 1100), (64, False, 1100), (128, True, 1100)])
def test_table_gradient_of_a_crowded_bucket(d, causal, sk):
    """64 queries and many more keys: most keys share the last bucket, whose gradient is what is left of near-equal
    sums.  delta comes from outputs rounded to 16 bits, so that its error, up to 2^-9 |O| |dO| in a row, stands
    there times the row's probability of the bucket, with nothing to cancel against: the rows' errors add up
    like a random walk (twice that allowed) to the rounding of the terms, as everywhere."""
    b, sq, h = 2, 64, 3
    torch.manual_seed(d)
    q, k, v = (torch.randn(b, n, h, d, device="cuda", dtype=torch.bfloat16, requires_grad=True) for n in (sq, sk, sk))
    table = (torch.randn(32, h, device="cuda") * 0.5).requires_grad_(True)
    out = NF.flash_attention(q, k, v, causal=causal, rel_bias_table=table, rel_bidirectional=not causal)
    g = torch.randn_like(out)
    (got,) = torch.autograd.grad(out, [table], g)
    want_out, _, _, _, leaf = _reference(q, k, v, None, causal, d ** -0.5, table, None, 0.0)
    (want,) = torch.autograd.grad(want_out, [leaf], g.double())
    pos = torch.arange(sk, device="cuda")[None] - (torch.arange(sq, device="cuda")[:, None] + sk - sq)
    buckets = NF.t5_relative_position_bucket(pos, not causal, 32, 128)
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * d ** -0.5 + table.double()[buckets].permute(2, 0, 1)
    if causal:
        s = s.masked_fill(torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1), float("-inf"))
    mass = torch.einsum("bhqk,qkn->bhqn", torch.softmax(s, -1), torch.nn.functional.one_hot(buckets, 32).double())
    row = 2.0 ** -9 * (want_out.norm(dim=-1) * g.double().norm(dim=-1)).transpose(1, 2)       # [b, h, q]
    bound = 2 * (row[..., None] * mass).square().sum((0, 2)).sqrt().t()                       # [bucket, h]
    assert (got.double() - want).norm() < bound.norm() + TOL[torch.bfloat16] * want.norm()
    assert native.ops().device_status() == 0


# more work items than CTAs, of one and of an odd number of half tiles: a group's turn moves from
# item to item
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("sq,sk", [(60, 60), (150, 150)])
def test_turns_over_items(sq, sk, d):
    _check(40, sq, sk, 8, d, torch.bfloat16, "", 0.1)
