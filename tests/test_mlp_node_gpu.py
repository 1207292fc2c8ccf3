"""The feed-forward block's autograd node under what its layers had to bear: saved-tensor hooks, inputs that
are differentiated alone, and transforms, which are refused with the reason whatever they batch."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from slapo_b200.op import FusedMLP
from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _block(act, p):
    torch.manual_seed(2)
    block = FusedMLP(64, 256, act, p, device="cuda", dtype=BF)
    x = torch.randn(40, 64, device="cuda", dtype=BF, requires_grad=True)
    return block, x, [x, *block.parameters()]


def _run(block, x):
    torch.cuda.manual_seed(7)
    return block(x)


@pytest.mark.parametrize("act,p", [("gelu", 0.1), ("relu", 0.0)])
def test_hooks_and_single_inputs(act, p):
    block, x, leaves = _block(act, p)
    y = _run(block, x)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(1), t.cpu())[1], lambda t: t.cuda()):
        y = _run(block, x)
    assert seen and all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, leaves, dy), want))
    for i, leaf in enumerate(leaves):
        for other in leaves:
            other.requires_grad_(other is leaf)
        (got,) = torch.autograd.grad(_run(block, x), [leaf], dy)
        assert torch.equal(got, want[i]), i


def test_transforms_are_refused():
    block, x, leaves = _block("gelu", 0.0)
    x = x.detach()
    names = [n for n, _ in block.named_parameters()]
    plain = [p.detach() for p in block.parameters()]
    with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        block(fwd.make_dual(x, torch.ones_like(x)))
    with pytest.raises(RuntimeError, match="functorch"):
        torch.vmap(block)(torch.stack([x, x]))
    for i, name in enumerate(names):        # each parameter batched, the biases among them
        def call(t):
            return torch.func.functional_call(block, {**dict(zip(names, plain)), name: t}, (x,))
        with pytest.raises(RuntimeError, match="functorch"):
            torch.vmap(call)(torch.stack([plain[i], plain[i]]))
    w, b = plain[:2]
    with pytest.raises(RuntimeError, match="functorch"):
        torch.vmap(lambda t: NF.linear(x, w, t, "gelu"))(torch.stack([b, b]))


@pytest.mark.parametrize("rows,n,k", [(17, 64, 64), (24, 16, 72), (128, 272, 64), (130, 48, 512),
                                      (257, 144, 136), (300, 1040, 128), (1000, 2064, 256), (2048, 512, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dropout_in_the_epilogue(rows, n, k, dtype):
    """To the bit what a product followed by bias and dropout gives, in every tile that a product can get."""
    torch.manual_seed(rows + n)
    ops = native.ops()
    a = torch.randn(rows, k, device="cuda", dtype=dtype)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)
    for bias in (None, torch.randn(n, device="cuda", dtype=dtype)):
        for p in (0.1, 0.5):
            rng = ops.philox_reserve(rows * n)
            got = ops.gemm_dropout_fwd(a, w, bias, p, rng)
            want = ops.bias_dropout_add_fwd(ops.gemm(a, w, None, -1, False, False), bias, None, p, rng)
            assert torch.equal(got, want)
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,n,k,tile", [
    (4100, 2576, 128, (True, 0)), (16384, 1024, 64, (True, 0)), (2049, 4112, 72, (True, 0)),
    (1000, 2064, 136, (True, 128)), (120, 148 * 64 + 16, 64, (False, 128)),
    (100, 148 * 128 + 48, 64, (False, 0)), (40, 144, 64, (False, 64))])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dropout_in_the_epilogue_of_each_tile(rows, n, k, tile, dtype):
    """As above, with the tile named: CTA pairs' of 256 and 128 columns, one CTA's of 64, 128 and 256, ragged
    last ones."""
    ops = native.ops()
    assert tuple(ops.gemm_tile(rows, n)) == tile
    torch.manual_seed(rows + n)
    a = torch.randn(rows, k, device="cuda", dtype=dtype)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)
    for bias in (None, torch.randn(n, device="cuda", dtype=dtype)):
        rng = ops.philox_reserve(rows * n)
        got = ops.gemm_dropout_fwd(a, w, bias, 0.1, rng)
        want = ops.bias_dropout_add_fwd(ops.gemm(a, w, None, -1, False, False), bias, None, 0.1, rng)
        assert torch.equal(got, want)
    assert ops.device_status() == 0
