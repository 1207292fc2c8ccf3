"""Flash attention at the edges of its paths against a 64-bit restatement: work items beyond one
wave of the persistent grid, a single key tile, ragged and unequal lengths, keys split over work
items, row maxima that grow along the keys, relative bias and dropout on the general path.

Tolerance: P, dS and the results are rounded to 16 bits once each, an independent relative error of
up to 2^-9 (bf16) or 2^-12 (fp16) per value; the 2-norm of a result's error stays below four times
that."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native
from slapo_b200.ops.flash_attn import dropout_keep_mask, effective_dropout_p

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16
TOL = {BF: 4 * 2.0 ** -9, FP: 4 * 2.0 ** -12}


def _reference(q, k, v, bias, causal, scale, table, mask, p):
    q, k, v = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    sq, sk = s.shape[-2:]
    if table is not None:
        table = table.detach().double().requires_grad_(True)
        pos = torch.arange(sk, device="cuda")[None] - (torch.arange(sq, device="cuda")[:, None]
                                                       + sk - sq)
        s = s + table[NF.t5_relative_position_bucket(pos, not causal, 32, 128)].permute(2, 0, 1)
    if bias is not None:
        s = s + bias.double()[:, None, None]
    if causal:
        ahead = torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1)
        s = s.masked_fill(ahead, float("-inf"))
    pr = torch.softmax(s, -1).nan_to_num(nan=0.0)      # rows without a key give zeros
    if mask is not None:
        pr = pr * mask.double() / (1 - p)
    return torch.einsum("bhqk,bkhd->bqhd", pr, v), q, k, v, table


# batch, sq, sk, heads, dim, dtype, then: c causal, k key padding, r relative table, g growing
# scores; dropout probability
CASES = [
    (2, 512, 512, 40, 64, BF, "", 0.0),        # more row tiles than resident CTAs
    (1, 1024, 1024, 40, 128, FP, "", 0.0),
    (2, 640, 640, 30, 128, BF, "c", 0.1),
    (2, 300, 300, 3, 64, BF, "c", 0.0),
    (2, 200, 333, 3, 80, BF, "k", 0.0),
    (2, 333, 200, 3, 80, FP, "ck", 0.0),       # early queries see no key
    (2, 200, 333, 3, 64, BF, "c", 0.0),
    (3, 520, 520, 50, 64, FP, "k", 0.1),
    (300, 130, 130, 2, 64, BF, "", 0.1),
    (2, 256, 256, 4, 64, BF, "r", 0.0),
    (2, 200, 200, 4, 64, BF, "ckr", 0.1),
    (1, 300, 300, 4, 128, BF, "r", 0.1),
    (2, 130, 333, 3, 64, BF, "kr", 0.0),       # biases of ragged tiles and unequal lengths
    (1, 333, 130, 2, 80, FP, "r", 0.0),
    (20, 200, 300, 12, 64, FP, "kr", 0.0),     # ... of the next work item, fetched ahead
    (12, 260, 140, 9, 128, BF, "kr", 0.1),
    (2, 1024, 1024, 4, 64, BF, "g", 0.0),      # row maxima raised many times
    (2, 1024, 1024, 4, 128, FP, "cg", 0.1),
    (1, 1, 1000, 4, 128, BF, "c", 0.0),        # keys split over work items
    (3, 5, 700, 4, 64, BF, "ck", 0.0),
    (2, 100, 1500, 8, 80, FP, "g", 0.1),
    (8, 1, 1500, 16, 128, BF, "c", 0.0),
    (1, 48, 2048, 4, 40, BF, "cr", 0.1),
    (1, 400, 1700, 2, 64, BF, "c", 0.1),       # dQ: keys split, some splits beyond the diagonal
    (2, 400, 1700, 2, 128, FP, "ck", 0.0),
    (1, 1700, 100, 6, 128, BF, "", 0.1),       # passes of unequal lengths side by side
    (9, 256, 256, 16, 64, FP, "c", 0.0),       # ... of several work items per CTA
    (6, 256, 256, 16, 128, BF, "k", 0.1),
    (20, 130, 130, 16, 64, BF, "", 0.1),
    (1, 1, 1, 1, 8, BF, "", 0.0),
    (2, 129, 1, 2, 64, BF, "", 0.0),
]


@pytest.mark.parametrize("b,sq,sk,h,d,dtype,how,p", CASES)
def test_flash_attention_paths(b, sq, sk, h, d, dtype, how, p):
    torch.manual_seed(b + sq + sk + h + d)
    q = torch.randn(b, sq, h, d, device="cuda", dtype=dtype, requires_grad=True)
    k = torch.randn(b, sk, h, d, device="cuda", dtype=dtype)
    if "g" in how:
        k = (k * torch.linspace(0.2, 6, sk, device="cuda")[None, :, None, None]).to(dtype)
    k.requires_grad_(True)
    v = torch.randn(b, sk, h, d, device="cuda", dtype=dtype, requires_grad=True)
    bias = None
    if "k" in how:
        # at least half of the keys are real: with a handful dS = P (dP - delta) cancels, and its
        # error, 2^-9 P (|dP| + |delta|), is bounded against the terms but not against dS
        real = torch.randint((sk + 1) // 2, sk + 1, (b, 1), device="cuda")
        bias = torch.where(torch.arange(sk, device="cuda")[None] < real, 0.0, -10000.0)
    table = (torch.randn(32, h, device="cuda") * 0.5).requires_grad_(True) if "r" in how else None
    causal = "c" in how
    torch.cuda.manual_seed(5)
    mask = dropout_keep_mask(b, h, sq, sk, p) if p else None
    out = NF.flash_attention(q, k, v, key_padding_bias=bias, causal=causal, dropout_p=p,
                             rel_bias_table=table, rel_bidirectional=not causal)
    g = torch.randn_like(out)
    out.backward(g)
    assert native.ops().device_status() == 0, "a bounded wait inside a kernel ran out"
    want, *leaves = _reference(q, k, v, bias, causal, d ** -0.5, table, mask,
                               effective_dropout_p(p))
    want.backward(g.double())
    got = [("out", out, want.detach())] + [
        (name, x.grad, y.grad) for name, x, y in zip(("dq", "dk", "dv", "dtable"),
                                                     (q, k, v, table), leaves) if x is not None]
    for name, x, y in got:
        # (with a single key dS is a difference of equal numbers: measured against unit scale)
        err = ((x.double() - y).norm() / y.norm().clamp(min=0.05 * y.numel() ** 0.5)).item()
        assert err < TOL[dtype], f"{name}: {err:.2e}"


@pytest.mark.parametrize("pairs", [1, 3])
@pytest.mark.parametrize("sq,sk,d,how", [(300, 200, 64, ""), (200, 300, 128, "ckr"), (130, 900, 64, "c")])
def test_backward_in_several_launches(sq, sk, d, how, pairs):
    """Keep bits of a few (batch, head) pairs at a time, the last launch with fewer: bit for bit
    what one launch for all of them gives (relative bias: sums of another order)."""
    torch.manual_seed(sq + sk)
    b, h, p = 2, 5, 0.1
    q, k, v = (torch.randn(b, n, h, d, device="cuda", dtype=BF) for n in (sq, sk, sk))
    bias = torch.zeros(b, sk, device="cuda").masked_fill(
        torch.arange(sk, device="cuda") >= sk - 20, -10000.0) if "k" in how else None
    rel = torch.randn(h, sq + sk - 1, device="cuda") if "r" in how else None
    ops, causal = native.ops(), "c" in how
    rng = ops.philox_reserve(b * h * sq * sk)
    out, lse = ops.flash_attn_fwd(q, k, v, bias, rel, causal, d ** -0.5, p, rng)
    dout = torch.randn_like(out)
    words = (-(-sk // 128) * 4) * (-(-sq // 128) * 128)

    def backward(n):
        before = native.launch_count()
        got = ops.flash_attn_bwd(dout, q, k, v, out, lse, bias, rel, causal, d ** -0.5, p, rng, False,
                                 n * words)
        return got, native.launch_count() - before

    few, n_few = backward(pairs)
    every, n_every = backward(b * h)
    assert n_few - n_every == 2 * (-(-b * h // pairs) - 1)
    assert all(torch.equal(x, y) for x, y in zip(few[:3], every[:3]))
    torch.testing.assert_close(few[3], every[3], rtol=1e-4, atol=1e-4)
    drawn, _ = backward(0)               # the passes side by side draw the same decisions
    assert all(torch.equal(x, y) for x, y in zip(drawn[:3], every[:3]))
    assert native.ops().device_status() == 0


@pytest.mark.parametrize("b,sq,sk", [(1, 0, 700), (1, 700, 0), (0, 64, 64), (65536, 1, 1)])
def test_empty_and_oversized_calls_are_refused(b, sq, sk):
    q, k = (torch.zeros(b, n, 2, 64, device="cuda", dtype=BF) for n in (sq, sk))
    lse = torch.zeros(b, 2, sq, device="cuda")
    if q.numel() == 0 or k.numel() == 0:
        with pytest.raises(RuntimeError, match="refused"):
            native.ops().flash_attn_fwd(q, k, k, None, None, False, 0.125, 0.0, None)
    with pytest.raises(RuntimeError, match="refused"):
        native.ops().flash_attn_bwd(q, q, k, k, q, lse, None, None, False, 0.125, 0.1,
                                    native.ops().philox_reserve(8), False)


@pytest.mark.parametrize("bh,sk,d,launches", [
    (128, 1500, 128, 1),      # one CTA per SM: a second item per head would wait for the first
    (128, 1500, 64, 2),       # two per SM
    (12, 1500, 128, 2),
    (12, 300, 64, 1),         # too few tiles to shorten
    (300, 4000, 64, 1),
])
def test_keys_are_split_where_that_shortens_the_chain(bh, sk, d, launches):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule counts SMs")
    q, k, v = (torch.randn(1, n, bh, d, device="cuda", dtype=BF) for n in (1, sk, sk))
    before = native.launch_count()
    NF.flash_attention(q, k, v)
    assert native.launch_count() - before == launches


def _rounded_as_the_running_maximum_says(q, k, v, scale, dtype, tile=128):
    """64-bit attention with one rounding of P, scaled by the row maximum of the keys up to and
    including its tile, and one of the result: what the order of an online softmax gives."""
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * scale
    v = v.double().transpose(1, 2)
    m = torch.full(s.shape[:-1], float("-inf"), device=s.device, dtype=s.dtype)
    o, l = torch.zeros_like(q.double().transpose(1, 2)), torch.zeros_like(m)
    for at in range(0, s.shape[-1], tile):
        part = s[..., at:at + tile]
        new = torch.maximum(m, part.amax(-1))
        p = torch.exp(part - new[..., None])
        shrink = torch.exp(m - new)
        o = o * shrink[..., None] + p.to(dtype).double() @ v[..., at:at + tile, :]
        l = l * shrink + p.sum(-1)
        m = new
    return (o / l[..., None]).to(dtype).transpose(1, 2)


@pytest.mark.parametrize("sk,d,dtype,grow", [(512, 64, BF, False), (1024, 128, BF, False),
                                             (512, 64, FP, False), (1024, 64, BF, True)])
def test_forward_rounds_no_more_than_an_online_softmax(sk, d, dtype, grow):
    """P scaled by an older maximum lies anywhere in its binade and is rounded more coarsely where
    it counts (5 % of the result's error at 512 keys); half a million results put the two errors'
    ratio within 0.3 %."""
    torch.manual_seed(sk + d)
    q, k, v = (torch.randn(4, n, 4, d, device="cuda", dtype=dtype) for n in (512, sk, sk))
    if grow:
        k = (k * torch.linspace(0.5, 2, sk, device="cuda")[None, :, None, None]).to(dtype)
    scale = d ** -0.5
    want = _reference(q, k, v, None, False, scale, None, None, 0.0)[0].detach()
    got = NF.flash_attention(q, k, v)
    err = [((x.double() - want).norm() / want.norm()).item()
           for x in (got, _rounded_as_the_running_maximum_says(q, k, v, scale, dtype))]
    assert err[0] < 1.01 * err[1], err
