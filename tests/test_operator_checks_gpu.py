"""What the GEMM's epilogue operators take and refuse: biases that are missing, start off a 16-byte boundary,
lie elsewhere or have another length.  (None of these may reach a kernel that would read out of range.)"""
import pytest
import torch
import torch.nn.functional as F

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _inputs(m, k, n):
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda", dtype=BF, requires_grad=True)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(BF).requires_grad_()
    return x, w, torch.randn(n + 8, device="cuda", dtype=BF)


# rows for the few-rows kernel, one CTA per tile, pairs
@pytest.mark.parametrize("m", [8, 40, 392])
@pytest.mark.parametrize("act", ["gelu", "relu", None])
@pytest.mark.parametrize("how", ["none", "odd"])
def test_bias_missing_or_unaligned(m, act, how):
    x, w, b = _inputs(m, 64, 4104)
    b = None if how == "none" else b[1:4105].detach().requires_grad_()
    code = -1 if act is None else NF._act_code(act)
    y = native.ops().linear(x, w, b, code, False)
    leaves = [t for t in (x, w, b) if t is not None]
    got = torch.autograd.grad(y.sum(), leaves)
    exact = [t.detach().double().requires_grad_() for t in leaves]
    want = F.linear(exact[0], exact[1], exact[2] if b is not None else None)
    want = {"gelu": F.gelu, "relu": F.relu, None: lambda t: t}[act](want)
    for p, q in zip([y, *got], [want, *torch.autograd.grad(want.sum(), exact)]):
        # four roundings to bf16
        assert ((p.double() - q).norm() / q.norm()).item() < 4 * 2.0 ** -9
    if act is not None:      # the front end's own way round
        assert torch.equal(NF.linear(x, w, b, act), y)


def test_block_with_unaligned_biases():
    x, w1, b = _inputs(40, 64, 256)
    w2 = (torch.randn(64, 256, device="cuda") / 16).to(BF).requires_grad_()
    b1, b2 = b[1:257], b[3:67]
    want = F.linear(F.gelu(F.linear(x, w1, b1).float()).to(BF), w2, b2)
    for p in (0.0, 0.5):
        y = native.ops().mlp(x, w1, b1, w2, b2, 0, p)
        kept = (y != 0) if p else torch.ones_like(y, dtype=torch.bool)
        assert ((y * (1 - p) - want)[kept].norm() / want.norm()).item() < 4 * 2.0 ** -9


def test_refusals():
    ops = native.ops()
    x, w, b = _inputs(392, 64, 4104)
    for bias in (b[:4104].cpu(), b[:4096], b[:4104].float()):
        for call in (lambda: ops.gemm_act_fwd(x, w, bias, 0, False),
                     lambda: ops.gemm(x, w, bias, -1, False, False),
                     lambda: ops.linear(x, w, bias, 0, False)):
            with pytest.raises(RuntimeError):
                call()
    with pytest.raises(RuntimeError):
        ops.gemm_act_fwd(x, w, b[1:4105], 0, False)
    with pytest.raises(RuntimeError):
        ops.gemm(x, w.detach().cpu(), None, -1, False, False)
    w2 = torch.zeros(64, 4104, device="cuda", dtype=BF)
    good = (x, w, b[:4104], w2, b[:64])
    ops.mlp(*good, 0, 0.0)
    for i, t in ((1, w[:, :56]), (2, b[:4096]), (2, b[:4104].cpu()), (3, w2[:, :4096]), (3, w2.cpu()),
                 (4, b[:56]), (4, b[:64].cpu()), (4, b[:64].float())):
        bad = list(good)
        bad[i] = t
        for p in (0.0, 0.5):
            with pytest.raises(RuntimeError):
                ops.mlp(*bad, 0, p)
    for bias in (b[:64].cpu(), b[1:65]):
        with pytest.raises(RuntimeError):
            ops.bias_act_fwd(x, bias, 0)
    assert ops.device_status() == 0
