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


@pytest.mark.parametrize("d,causal,sk", [(64, True, 700), (64, True, 1100), (64, False, 1100),
                                         (128, True, 1100)])
def test_table_gradient_of_a_crowded_bucket(d, causal, sk):
    """64 queries and many more keys: most keys share the last bucket, whose gradient is what is left of
    near-equal sums.  delta comes from outputs rounded to 16 bits, so that its error, up to 2^-9 |O| |dO| in a
    row, stands there times the row's probability of the bucket, with nothing to cancel against: the rows'
    errors add up like a random walk (twice that allowed) to the rounding of the terms, as everywhere."""
    b, sq, h = 2, 64, 3
    torch.manual_seed(d)
    q, k, v = (torch.randn(b, n, h, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
               for n in (sq, sk, sk))
    table = (torch.randn(32, h, device="cuda") * 0.5).requires_grad_(True)
    out = NF.flash_attention(q, k, v, causal=causal, rel_bias_table=table, rel_bidirectional=not causal)
    g = torch.randn_like(out)
    (got,) = torch.autograd.grad(out, [table], g)
    want_out, _, _, _, leaf = _reference(q, k, v, None, causal, d ** -0.5, table, None, 0.0)
    (want,) = torch.autograd.grad(want_out, [leaf], g.double())
    pos = torch.arange(sk, device="cuda")[None] - (torch.arange(sq, device="cuda")[:, None] + sk - sq)
    buckets = NF.t5_relative_position_bucket(pos, not causal, 32, 128)
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * d ** -0.5
    s = s + table.double()[buckets].permute(2, 0, 1)
    if causal:
        s = s.masked_fill(torch.ones_like(s[0, 0], dtype=torch.bool).triu(sk - sq + 1), float("-inf"))
    mass = torch.einsum("bhqk,qkn->bhqn", torch.softmax(s, -1),
                        torch.nn.functional.one_hot(buckets, 32).double())
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


# Every CTA's first item, all loads of the launch at once: products must not run ahead of the tiles that
# they read.
@pytest.mark.parametrize("b,sq,sk,h,d,causal", [(36, 256, 15, 16, 128, False), (32, 672, 12, 16, 128, False),
                                                (39, 642, 288, 8, 128, True), (14, 1039, 186, 16, 96, True),
                                                (39, 256, 256, 16, 128, False), (60, 256, 40, 16, 64, False)])
def test_first_items_of_a_launch(b, sq, sk, h, d, causal):
    torch.manual_seed(sq + sk)
    q, k, v, g = (torch.randn(b, n, h, d, device="cuda", dtype=torch.bfloat16) for n in (sq, sk, sk, sq))
    ops = native.ops()
    out, lse = ops.flash_attn_fwd(q, k, v, None, None, causal, d ** -0.5, 0.0, None)
    once = ops.flash_attn_bwd(g, q, k, v, out, lse, None, None, causal, d ** -0.5, 0.0, None, False)[:3]
    for _ in range(6):
        again = ops.flash_attn_bwd(g, q, k, v, out, lse, None, None, causal, d ** -0.5, 0.0, None, False)
        assert all(torch.equal(x, y) for x, y in zip(again, once))      # (sums have one order)
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * d ** -0.5
    if causal:
        s = s.masked_fill(torch.ones_like(s[0, 0], dtype=torch.bool).triu(sk - sq + 1), float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)
    dv = torch.einsum("bhqk,bqhd->bkhd", p, g.float())
    ds = p * (torch.einsum("bqhd,bkhd->bhqk", g.float(), v.float())
              - (g.float() * out.float()).sum(-1).transpose(1, 2)[..., None])
    dk = torch.einsum("bhqk,bqhd->bkhd", ds, q.float()) * d ** -0.5
    dq = torch.einsum("bhqk,bkhd->bqhd", ds, k.float()) * d ** -0.5
    for got, want in zip(once, (dq, dk, dv)):
        # each head of its own: a single wrong half tile shows
        err = (got.float() - want).square().sum((1, 3)).sqrt() / want.square().sum((1, 3)).sqrt()
        assert err.max().item() < 2 * TOL[torch.bfloat16]
    assert ops.device_status() == 0
