"""Small kernels and dispatch rules at the sizes where they can go wrong."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native
from slapo_b200.ops.flash_attn import relative_bias_by_distance

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (1, 72, 64, False, False),
    (128, 64 * 148, 64, False, False),     # the last width with one wave of 64-column tiles
    (128, 64 * 148 + 8, 64, False, True),
    (128, 128 * 148 + 8, 64, False, False),
    (129, 64, 72, False, True),
    (200, 768, 2048, False, False),        # narrow tiles, whatever the contraction
    (200, 768, 2056, False, True),
    (384, 4096, 1024, False, False),       # 128-column pairs
    (520, 9216, 136, False, False),        # beyond one wave of them
    (768, 776, 8, True, True),
    (264, 136, 200, True, False),
])
def test_gemm_tile_choice(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", dtype=BF)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", dtype=BF)
    bias = torch.randn(N, device="cuda", dtype=BF)
    c = native.ops().gemm_out(a, b, bias, 2, a_mn, b_mn, None, None, 0, False)
    assert native.ops().device_status() == 0
    want = torch.relu((a.double().t() if a_mn else a.double())
                      @ (b.double() if b_mn else b.double().t()) + bias.double())
    # fp32 sums, one rounding to bf16
    assert ((c.double() - want).norm() / want.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("dtype", [BF, FP, torch.float32])
@pytest.mark.parametrize("b,past,new,h,d", [(1, 1, 1, 1, 8), (3, 130, 5, 4, 64), (2, 0, 3, 2, 80),
                                            (5, 777, 1, 3, 128)])
def test_kv_append(dtype, b, past, new, h, d):
    pk, pv = (torch.randn(b, past, h, d, device="cuda", dtype=dtype) for _ in range(2))
    qkv = torch.randn(b, new, h, 3, d, device="cuda", dtype=dtype)
    k, v = qkv[..., 1, :], qkv[..., 2, :]
    before = native.launch_count()
    got = NF.append_kv(pk, pv, k, v)
    assert native.launch_count() == before + 1
    for x, p, n in zip(got, (pk, pv), (k, v)):
        want = torch.cat((p, n), dim=1)
        assert x.stride() == want.stride() and torch.equal(x, want)


def test_kv_append_leaves_other_inputs_to_cat():
    k = torch.randn(2, 3, 2, 64, device="cuda", dtype=BF)
    past = torch.randn(2, 9, 2, 64, device="cuda", dtype=BF, requires_grad=True)
    before = native.launch_count()
    out, _ = NF.append_kv(past, past, k, k)                       # a gradient is wanted
    assert out.requires_grad
    NF.append_kv(past.detach().transpose(1, 2).contiguous().transpose(1, 2), past.detach(), k, k)
    NF.append_kv(past.detach()[..., :4], past.detach()[..., :4], k[..., :4], k[..., :4])
    NF.append_kv(past.detach().float(), past.detach(), k, k)      # types differ
    NF.append_kv(past.detach(), past.detach(), k.expand(2, 3, 2, 64)[:, :0], k[:, :0])
    stacked = torch.stack([k, -k])
    got = torch.vmap(lambda t: NF.append_kv(past.detach(), past.detach(), t, t)[0])(stacked)
    assert torch.equal(got[1], torch.cat((past.detach(), -k), dim=1))
    out, dot = torch.func.jvp(lambda t: NF.append_kv(past.detach(), t, k, k)[1], (past.detach(),),
                              (past.detach(),))
    assert torch.equal(dot[:, :9], past.detach()) and (dot[:, 9:] == 0).all()
    with torch.no_grad(), torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(k, k)
        out = torch.autograd.forward_ad.unpack_dual(NF.append_kv(past, past, dual, k)[0])
        assert torch.equal(out.tangent[:, 9:], k)
    assert native.launch_count() == before
    NF.append_kv(past.detach(), past.detach(), k, k)
    with torch.no_grad():
        NF.append_kv(past, past, k, k)
    assert native.launch_count() == before + 2


@pytest.mark.parametrize("dtype", [torch.float32, BF, FP])
@pytest.mark.parametrize("buckets,heads,sq,sk", [(32, 3, 1, 1), (32, 16, 200, 200), (8, 1, 5, 300)])
def test_relative_bias(dtype, buckets, heads, sq, sk):
    table = torch.randn(buckets, heads, device="cuda", dtype=dtype, requires_grad=True)
    out = relative_bias_by_distance(table, sq, sk, True, 128)
    dist = torch.arange(-(sq - 1), sk, device="cuda") - (sk - sq)
    at = NF.t5_relative_position_bucket(dist, True, buckets, 128)
    assert torch.equal(out, table.detach().float()[at].t())
    g = torch.randn_like(out)
    out.backward(g)
    want = torch.zeros(buckets, heads, device="cuda", dtype=torch.float64)
    want.index_add_(0, at, g.t().double())
    # fp32 sums of up to sq + sk - 1 terms, rounded once to the table's type
    eps = {torch.float32: 2.0 ** -18, BF: 2.0 ** -8, FP: 2.0 ** -11}[dtype]
    assert ((table.grad.double() - want).norm() / want.norm()).item() < eps


def test_relative_bias_under_transforms():
    """What indexing the table could do: second derivatives, forward mode, vmap."""
    sq, sk = 20, 33
    table = torch.randn(32, 3, device="cuda", requires_grad=True)

    def by_indexing(t):
        dist = torch.arange(-(sq - 1), sk, device="cuda") - (sk - sq)
        return t.float()[NF.t5_relative_position_bucket(dist, True, 32, 128)].t()

    def bias(t):
        return relative_bias_by_distance(t, sq, sk, True, 128)

    grads = []
    for fn in (bias, by_indexing):
        (g,) = torch.autograd.grad((fn(table) ** 3).sum(), table, create_graph=True)
        grads.append(torch.autograd.grad((g ** 2).sum(), table)[0])
    torch.testing.assert_close(*grads)
    v = torch.randn_like(table)
    for got, want in zip(torch.func.jvp(bias, (table.detach(),), (v,)),
                         torch.func.jvp(by_indexing, (table.detach(),), (v,))):
        assert torch.equal(got, want)
    assert torch.equal(torch.vmap(bias)(torch.stack([v, -v])), torch.stack([bias(v), bias(-v)]))


def test_relative_bias_refuses_what_does_not_fit():
    ops = native.ops()
    table = torch.randn(8, 3, device="cuda")
    at = torch.arange(5, device="cuda")
    grad = torch.randn(3, 5, device="cuda")
    for args in ((table, at.int()), (table, at.cpu()), (table, at[None]), (table.double(), at),
                 (table.t(), at), (table[0], at)):
        with pytest.raises(RuntimeError):
            ops.rel_bias_fwd(*args)
    for args in ((grad, at.int(), table), (grad, at.cpu(), table), (grad[:, :4], at, table),
                 (grad[:2], at, table), (grad.t(), at, table), (grad.half(), at, table),
                 (grad[0], at, table), (grad, at, table.double()), (grad, at, table[0]),
                 (grad, at[:4], table), (grad.cpu(), at, table)):
        with pytest.raises(RuntimeError):
            ops.rel_bias_bwd(*args)


def test_relative_bias_indexes_outside_of_the_table():
    """Negative ones count from the end; what lies outside is not read: NaN, and no gradient."""
    ops = native.ops()
    table = torch.randn(4, 2, device="cuda")
    at = torch.tensor([-1, 3, 4, -5, 0, 1 << 40], device="cuda")
    out = ops.rel_bias_fwd(table, at)
    assert torch.equal(out[:, [0, 1, 4]], table.t()[:, [3, 3, 0]])
    assert out[:, [2, 3, 5]].isnan().all()
    grad = torch.ones(2, 6, device="cuda")
    want = torch.tensor([1.0, 0, 0, 2], device="cuda")[:, None].expand(4, 2)
    assert torch.equal(ops.rel_bias_bwd(grad, at, table), want)


@pytest.mark.parametrize("dtype", [BF, FP])
def test_gelu_extremes(dtype):
    big = 60000.0 if dtype == FP else 1e30
    x = torch.tensor([float("inf"), float("nan"), big, -big, 0.0, -0.0, 12.0, -12.0] * 4,
                     device="cuda", dtype=dtype).view(4, 8)
    y = NF.bias_act(x, None, "gelu")
    assert y[0, 0] == float("inf") and y[0, 1].isnan() and y[0, 2] == x[0, 2]
    assert y[0, 3] == 0 and (y[0, 4:6] == 0).all() and y[0, 6] == 12 and y[0, 7].abs() < 1e-6


def test_dropout_add_norm_outputs_without_a_consumer():
    x, r = (torch.randn(5, 64, device="cuda", dtype=BF, requires_grad=True) for _ in range(2))
    w, b = (torch.randn(64, device="cuda", dtype=BF, requires_grad=True) for _ in range(2))
    for pick in ((0,), (1,), (0, 1)):
        out = NF.dropout_add_layer_norm(x, None, r, w, b, 0.0, 1e-5, True)
        xf, rf, wf, bf = (t.detach().double().requires_grad_(True) for t in (x, r, w, b))
        z = xf + rf
        ref = (torch.nn.functional.layer_norm(z, (64,), wf, bf, 1e-5), z)
        got = torch.autograd.grad([out[i].float().sum() * (i + 1) for i in pick], [x, r, w, b],
                                  allow_unused=True)
        want = torch.autograd.grad([ref[i].sum() * (i + 1) for i in pick], [xf, rf, wf, bf],
                                   allow_unused=True)
        for g, t in zip(got, want):
            t = torch.zeros_like(g, dtype=torch.float64) if t is None else t
            scale = t.norm().clamp(min=t.numel() ** 0.5)
            assert ((g.double() - t).norm() / scale).item() < 2.0 ** -6
