"""Loss and log-sum-exp of unsharded logits from one kernel: columns around its unrolled step (four times
256 threads of 8), ignored rows, labels outside of the vocabulary and hidden logits."""
import pytest
import torch

from slapo_b200.ops import cross_entropy as ce
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (5, 2040), (3, 2056), (4, 8192), (7, 8200), (2, 50304)])
def test_loss_and_gradient(rows, cols, dtype):
    torch.manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda") * 3).to(dtype)
    if cols > 64:
        x[0, 8:cols // 2] = float("-inf")        # whole vectors of a thread among them
    labels = torch.randint(0, 8, (rows,), device="cuda")
    if rows > 2:
        labels[1] = -100
    x.requires_grad_()
    loss = ce.cross_entropy(x, labels)
    coef = torch.rand(rows, device="cuda")
    loss.backward(coef)
    want = torch.nn.functional.cross_entropy(x.detach().double(), labels, reduction="none",
                                             ignore_index=-100)
    # fp32: one rounding of sums of up to 50304 terms, which exp2's own 2e-7 relative dominates
    torch.testing.assert_close(loss.double(), want, rtol=2e-6, atol=2e-6)
    p = torch.softmax(x.detach().double(), -1)
    p[torch.arange(rows, device="cuda"), labels.clamp(min=0)] -= 1
    p = p * (coef.double() * (labels != -100))[:, None]
    err = ((x.grad.double() - p).norm() / p.norm()).item()
    assert err < {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10, torch.float32: 5e-6}[dtype]


@pytest.mark.parametrize("cols", [16376, 16384, 16392])      # a vector at a time, and four
def test_border_of_long_rows(cols):
    torch.manual_seed(cols)
    x = torch.randn(9, cols, device="cuda").bfloat16()
    labels = torch.randint(0, cols, (9,), device="cuda")
    labels[4] = -100
    loss, lse = native.ops().ce_loss(x, labels, -100)
    stats = native.ops().ce_stats(x, labels, 0, -100).double()
    want = torch.logsumexp(x.double(), -1) * (labels != -100)
    picked = x.double()[torch.arange(9, device="cuda"), labels.clamp(min=0)] * (labels != -100)
    torch.testing.assert_close(lse.double(), want, rtol=2e-6, atol=2e-6)
    torch.testing.assert_close(loss.double(), want - picked, rtol=2e-6, atol=2e-6)
    ok = labels != -100
    torch.testing.assert_close((stats[:, 0] + stats[:, 1].log())[ok], want[ok], rtol=2e-6, atol=2e-6)
    assert torch.equal(stats[:, 2], picked) and stats[4].tolist() == [float("-inf"), 0.0, 0.0]


def test_error_of_peaked_rows():
    """A trained model's rows: logits spread over 40, a handful of terms make the sum."""
    torch.manual_seed(5)
    x = (torch.randn(512, 49152, device="cuda") * 5).bfloat16()
    labels = torch.randint(0, x.shape[1], (x.shape[0],), device="cuda")
    _, lse = native.ops().ce_loss(x, labels, -100)
    want = torch.logsumexp(x.double(), -1)
    # the result's own rounding to 32 bits, and 2^-20 for the terms (exp2: 2^-22) and their sum
    ulp = 2.0 ** (want.abs().log2().floor() - 23)
    assert ((lse.double() - want).abs() <= ulp / 2 + 2.0 ** -20).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("cols", [520, 8192, 50304])
def test_columns_masked_with_the_lowest_value(cols, dtype):
    torch.manual_seed(cols)
    low = torch.finfo(dtype).min
    x = torch.randn(4, cols, device="cuda").to(dtype)
    x[0, :cols - 8] = low               # all that most threads see
    x[1, :cols // 2] = low
    x[2, cols // 2:] = low
    x[3, 0] = -low
    labels = torch.tensor([cols - 3, cols - 1, 1, 0], device="cuda")
    x.requires_grad_()
    loss = ce.cross_entropy(x, labels)
    want = torch.nn.functional.cross_entropy(x.detach().double(), labels, reduction="none")
    torch.testing.assert_close(loss.double(), want, rtol=2e-6, atol=2e-6)
    (grad,) = torch.autograd.grad(loss.sum(), [x])
    p = torch.softmax(x.detach().double(), -1)
    p[torch.arange(4, device="cuda"), labels] -= 1
    torch.testing.assert_close(grad.double(), p, rtol=2.0 ** -7, atol=1e-6)
