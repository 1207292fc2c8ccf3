"""Activations and their derivatives in the GEMM's epilogue at the edges of its tiles, against 64 bits,
and the feed-forward block as one node against its two layers."""
import pytest
import torch
import torch.nn.functional as F

from slapo_b200.op import FusedMLP
from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16
# one rounding of each value to 16 bits, up to 2^-9 (bf16) or 2^-12 (fp16) relative, four times over
TOL = {BF: 4 * 2.0 ** -9, FP: 4 * 2.0 ** -12}


def _act(x, name):
    if name == "relu":
        return F.relu(x)
    return F.gelu(x, approximate="none" if name == "gelu" else "tanh")


def _close(got, want, tol):
    return ((got.double() - want).norm() / want.norm().clamp(min=1e-30)).item() < tol


# rows, inner, columns: one narrow tile; a ragged one of each kind (single CTA of 64 / 128 / 256 columns,
# pairs of 128 / 256); several row blocks and work items
SHAPES = [(8, 64, 8), (40, 72, 200), (128, 64, 4096), (120, 64, 19200), (136, 264, 136), (264, 64, 72),
          (200, 3072, 768), (1000, 2560, 1096), (2056, 64, 2056), (33 * 8, 8, 24)]


@pytest.mark.parametrize("act,dtype", [("gelu", BF), ("gelu_new", FP), ("relu", BF)])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_epilogue(m, k, n, act, dtype):
    torch.manual_seed(m + k + n)
    x = torch.randn(m, k, device="cuda", dtype=dtype)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)
    b = torch.randn(n, device="cuda", dtype=dtype)
    z = F.linear(x.double(), w.double(), b.double())
    code = NF._act_code(act)
    ops = native.ops()
    if act != "relu":
        y, kept = ops.gemm_act_fwd(x, w, b, code, True)
        assert _close(y, _act(z, act), TOL[dtype]) and _close(kept, z, TOL[dtype])
        alone, none = ops.gemm_act_fwd(x, w, b, code, False)
        assert torch.equal(alone, y) and none.numel() == 0
        other = ops.linear(x, w.t().contiguous(), b, code, True)       # W as [in, out]
        assert _close(other, _act(z, act), TOL[dtype])
    # the derivative behind the following layer's input gradient: dy [m, k2] w2 [k2, n]
    dy = torch.randn(m, k, device="cuda", dtype=dtype)
    w2 = (torch.randn(k, n, device="cuda") * k ** -0.5).to(dtype)
    at = _act(z, act).to(dtype) if act == "relu" else z.to(dtype)
    zz = at.double().requires_grad_()
    (want,) = torch.autograd.grad(_act(zz, act), zz, dy.double() @ w2.double())
    dz, db = ops.gemm_act_bwd(dy, w2, at, code)
    assert _close(dz, want, TOL[dtype])
    assert _close(db, want.sum(0), TOL[dtype])
    assert ops.device_status() == 0


def test_epilogue_keeps_infinities_and_nans():
    x = torch.zeros(8, 64, device="cuda", dtype=BF)
    x[0, 0], x[1, 0], x[2, 0] = float("inf"), float("-inf"), float("nan")
    w = torch.ones(64, 64, device="cuda", dtype=BF)
    b = torch.zeros(64, device="cuda", dtype=BF)
    y, z = native.ops().gemm_act_fwd(x, w, b, 0, True)
    want = NF.bias_act(F.linear(x, w), b, "gelu")
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.isinf(y[0]).all()
    assert torch.isinf(z[:2]).all() and torch.isnan(z[2]).all() and (y[3:] == 0).all()


@pytest.mark.parametrize("tokens,hidden,act,p,dtype", [
    (8, 64, "gelu", 0.1, BF), (200, 256, "gelu_new", 0.1, FP), (1000, 512, "relu", 0.1, BF),
    (1032, 128, "relu", 0.0, FP), (264, 512, "gelu", 0.0, BF)])
def test_block_is_its_two_layers(tokens, hidden, act, p, dtype):
    """Same values, gradients and dropout mask as layer by layer, which a hook brings about."""
    torch.manual_seed(tokens)
    block = FusedMLP(hidden, 4 * hidden, act, p, device="cuda", dtype=dtype)
    x = torch.randn(2, tokens // 2, hidden, device="cuda", dtype=dtype, requires_grad=True)
    dy = torch.randn_like(x)
    leaves = [x, *block.parameters()]

    def run():
        torch.cuda.manual_seed(3)
        y = block(x)
        return [y, *torch.autograd.grad(y, leaves, dy)]

    one = run()
    before = native.launch_count()
    run()
    launches = native.launch_count() - before
    handle = block.fc_in.register_forward_hook(lambda m, i, o: None)
    two = run()
    handle.remove()
    assert ((one[0] == 0) == (two[0] == 0)).float().mean() > 0.999
    for a, b in zip(one, two):
        assert _close(a, b.double(), 2 * TOL[dtype])
    assert launches < 14
    # without gradients, and for some of the leaves only
    with torch.no_grad():
        torch.cuda.manual_seed(3)
        assert torch.equal(block(x), one[0])
    torch.cuda.manual_seed(3)
    (dw,) = torch.autograd.grad(block(x), [block.fc_out.weight], dy)
    assert torch.equal(dw, one[4])
    block.eval()
    assert _close(block(x), block.fc_out(block.fc_in(x)).double(), TOL[dtype])
