"""One token of generation at the edges of its kernels: attention of a single query, with and without
its keys split, and linear layers on up to 16 rows, against 64 bits."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native
from test_flash_paths_gpu import TOL, _reference

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16


@pytest.mark.parametrize("sk", [1, 31, 33, 128, 300, 1500, 4001])
@pytest.mark.parametrize("b,h,d,dtype,how", [(1, 4, 64, BF, ""), (2, 3, 128, FP, "c"), (3, 40, 80, BF, "k"),
                                             (300, 2, 8, FP, "ck"), (1, 12, 128, BF, "p")])
def test_single_query(sk, b, h, d, dtype, how):
    torch.manual_seed(sk + d)
    q = torch.randn(b, 1, h, d, device="cuda", dtype=dtype)
    if "p" in how:        # slices of a packed projection
        kv = torch.randn(b, sk, h, 3, d, device="cuda", dtype=dtype)
        k, v = kv[..., 1, :], kv[..., 2, :]
    else:
        k, v = (torch.randn(b, sk, h, d, device="cuda", dtype=dtype) for _ in range(2))
    bias = None
    if "k" in how:
        real = torch.randint((sk + 1) // 2, sk + 1, (b, 1), device="cuda")
        bias = torch.where(torch.arange(sk, device="cuda")[None] < real, 0.0, -10000.0)
    out = NF.flash_attention(q, k, v, key_padding_bias=bias, causal="c" in how)
    want = _reference(q, k, v, bias, "c" in how, d ** -0.5, None, None, 0.0)[0]
    assert ((out.double() - want).norm() / want.norm()).item() < TOL[dtype]
    # its gradients come from the same kernels as any other length's
    q.requires_grad_()
    NF.flash_attention(q, k, v, key_padding_bias=bias, causal="c" in how).sum().backward()
    wq = _reference(q, k, v, bias, "c" in how, d ** -0.5, None, None, 0.0)
    wq[0].sum().backward()
    assert (q.grad.double() - wq[1].grad).abs().max() < 0.05
    assert native.ops().device_status() == 0


# four warps per work item or sixteen: half a step of keys, two steps with 222 items, any number with 888
@pytest.mark.parametrize("h,sk,d", [(4, 128, 64), (4, 129, 64), (4, 64, 128), (4, 65, 80), (221, 512, 64),
                                    (222, 512, 64), (222, 513, 64), (222, 256, 128), (222, 257, 128),
                                     (887, 520, 64),
                                    (888, 520, 64), (888, 300, 128), (888, 7, 128)])
def test_warps_of_a_work_item(h, sk, d):
    test_single_query(sk, 1, h, d, BF, "k")


def test_keys_that_all_are_hidden():
    q, k, v = (torch.randn(1, n, 2, 64, device="cuda", dtype=BF) for n in (1, 200, 200))
    bias = torch.full((1, 200), float("-inf"), device="cuda")
    assert (NF.flash_attention(q, k, v, key_padding_bias=bias) == 0).all()


@pytest.mark.parametrize("sk", [40, 2000])        # one work item per head, and keys split
@pytest.mark.parametrize("what", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_nans_and_infinities_stay(sk, what, value):
    """An overflowed cache shows: what plain softmax attention makes a NaN or an infinity is one here, in its
    head, and the other heads are as they were."""
    torch.manual_seed(sk)
    q, k, v = (torch.randn(1, n, 3, 64, device="cuda", dtype=FP) for n in (1, sk, sk))
    clean = NF.flash_attention(q, k, v)
    {"q": q, "k": k, "v": v}[what][0, -1, 1, 5] = value
    out = NF.flash_attention(q, k, v)
    scores = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * 64 ** -0.5
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(scores, -1), v.double())
    assert torch.equal(out[:, :, [0, 2]], clean[:, :, [0, 2]])
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    if what == "v" or value != value:
        assert not out[:, :, 1].isfinite().all()


# steps of K in runs and one by one
@pytest.mark.parametrize("k", [2040, 2048, 2056, 4096, 4128, 768, 512])
def test_few_rows_contractions(k):
    test_few_rows(16, k, 1032, BF, None)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("k,n,dtype,act", [(64, 64, BF, None), (72, 200, FP, "relu"), (2048, 6144, BF, None),
                                           (2560, 72, FP, None), (4104, 1024, BF, "relu")])
def test_few_rows(m, k, n, dtype, act):
    torch.manual_seed(m + k)
    # rows of a wider tensor, as the last token of each sequence
    x = torch.randn(m, 2, k, device="cuda", dtype=dtype)[:, 1]
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)
    b = torch.randn(n, device="cuda", dtype=dtype)
    y = NF.linear(x, w, b, act)
    want = x.double() @ w.double().t() + b.double()
    want = want.relu() if act else want
    assert ((y.double() - want).norm() / want.norm()).item() < TOL[dtype]
    assert ((NF.linear(x, w).double() - x.double() @ w.double().t()).norm() / want.norm()).item() < TOL[dtype]
