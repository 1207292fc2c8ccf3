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


# rows, inner, columns, and the tile (of a CTA pair, its columns; 0: 256): narrow ones, a ragged one of each
# other kind, several row blocks and work items, more than one band of row tiles and a ragged last one
ONE64, ONE128, ONE256, PAIR128, PAIR256 = (False, 64), (False, 128), (False, 0), (True, 128), (True, 0)
SHAPES = [(8, 64, 8, ONE64), (40, 72, 200, ONE64), (128, 64, 4096, ONE64), (120, 64, 19200, ONE256),
          (136, 264, 136, ONE64), (264, 64, 72, ONE64), (200, 3072, 768, ONE64), (1000, 2560, 1096, ONE64),
          (2056, 64, 2056, PAIR256), (33 * 8, 8, 24, ONE64), (128, 64, 64 * 148 + 8, ONE128),
          (392, 64, 4104, PAIR128), (1000, 72, 2056, PAIR128), (2312, 72, 4360, PAIR256)]


@pytest.mark.parametrize("act,dtype", [("gelu", BF), ("gelu_new", FP), ("relu", BF)])
@pytest.mark.parametrize("m,k,n,tile", SHAPES)
def test_epilogue(m, k, n, tile, act, dtype):
    assert tuple(native.ops().gemm_tile(m, n)) == tile
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


@pytest.mark.parametrize("m,k,n,split", [
    (2312, 72, 4360, False),        # a band of eight row tiles and one of two, 18 column tiles
    (4104, 64, 4104, False),        # two whole bands and one of a ragged tile
    (264, 2048, 4360, True)])       # a band of two, two pairs per tile
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
def test_bands_of_row_tiles(m, k, n, split, a_mn, b_mn):
    torch.manual_seed(n)
    ops = native.ops()
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda", dtype=BF)
    w = torch.randn((k, n) if b_mn else (n, k), device="cuda", dtype=BF)
    b = torch.randn(n, device="cuda", dtype=BF)
    assert (ops.gemm2_splits(m, n, k) > 1) == split
    c = ops.gemm_out(a, w, b, -1, a_mn, b_mn, None, None, 0, split)
    want = (a.double().t() if a_mn else a.double()) @ (w.double() if b_mn else w.double().t()) + b.double()
    # each 128 x 128 block of its own: fp32 sums and one rounding
    err = (c.double() - want).square()
    for s, t in zip(err.split(128), want.square().split(128)):
        for p, q in zip(s.split(128, 1), t.split(128, 1)):
            assert (p.sum() / q.sum()).sqrt().item() < 2.0 ** -8
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
