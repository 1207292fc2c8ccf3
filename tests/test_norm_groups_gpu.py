"""Normalisation backward where its row groups and its one exchange of both sums can go wrong: fewer rows than
groups, a ragged last step, every width's thread layout, several rows per group one after the other."""
import pytest
import torch

from slapo_b200.ops import functional as NF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [8, 256, 264, 1024, 1032, 2048, 2056, 4096])
@pytest.mark.parametrize("rows", [1, 3, 5, 1186, 2375])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_gradients(rows, cols, rms):
    torch.manual_seed(rows + cols)
    x = torch.randn(rows, cols, device="cuda", requires_grad=True)
    w = (torch.rand(cols, device="cuda") + 0.5).requires_grad_()
    b = torch.randn(cols, device="cuda", requires_grad=True)
    dy = torch.randn(rows, cols, device="cuda")
    y = NF.rms_norm(x, w, 1e-6) if rms else NF.layer_norm(x, w, b, 1e-5)
    leaves = [x, w] if rms else [x, w, b]
    got = torch.autograd.grad(y, leaves, dy)
    again = torch.autograd.grad(NF.rms_norm(x, w, 1e-6) if rms else NF.layer_norm(x, w, b, 1e-5), leaves, dy)
    xx, ww, bb = (t.detach().double().requires_grad_() for t in (x, w, b))
    if rms:
        want = xx * torch.rsqrt(xx.square().mean(-1, keepdim=True) + 1e-6) * ww
    else:
        want = torch.nn.functional.layer_norm(xx, (cols,), ww, bb, 1e-5)
    ref = torch.autograd.grad(want, [xx, ww] if rms else [xx, ww, bb], dy.double())
    for a, c, r in zip(got, again, ref):
        # sums of up to 4096 values or 2375 rows in 32 bits: 2^-24 times the square root of their number,
        # a hundredfold
        assert (a.double() - r).norm() <= 4e-5 * r.norm() + 1e-6
        assert torch.equal(a, c)        # the sums have one order
