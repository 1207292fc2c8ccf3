"""Normalisation of 16-bit rows with 16 values per thread, against the general kernel (which takes the same
call with a weight that starts on 16 bytes only) and against 64 bits: every number of warps per row, its last
column group, fewer rows than groups, a ragged last step, and the numbers of rows from which the backward
takes the new form."""
import pytest
import torch

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu


def _off_32(t):
    room = torch.empty(t.numel() + 8, device="cuda", dtype=t.dtype)
    room[8:].copy_(t)
    return room[8:]


def _error(got, want):
    return float((got.double() - want).norm())


@pytest.mark.parametrize("cols", [272, 512, 528, 1024, 1040, 2048, 2064, 4096])
@pytest.mark.parametrize("rows", [1, 7, 4095, 6001])
@pytest.mark.parametrize("dtype,p", [(torch.bfloat16, 0.1), (torch.float16, 0.0), (torch.float16, 0.3)])
def test_sixteen_values_per_thread(rows, cols, dtype, p):
    ops = native.ops()
    torch.manual_seed(rows + cols)
    x, r, gy, gz = (torch.randn(rows, cols, device="cuda").to(dtype) for _ in range(4))
    bias, gamma, beta = (torch.randn(cols, device="cuda").to(dtype) for _ in range(3))
    rng = torch.tensor([77, 12, 0, 0], dtype=torch.int64) if p > 0 else None
    off = _off_32(gamma)
    assert gamma.data_ptr() % 32 == 0 and off.data_ptr() % 32 == 16
    new = ops.dropout_add_ln_fwd(x, bias, r, gamma, beta, p, 1e-5, rng)
    old = ops.dropout_add_ln_fwd(x, bias, r, off, beta, p, 1e-5, rng)
    assert torch.equal(new[1], old[1])                           # z: element by element, the same decisions
    y, z, mean, rstd = new
    back = ops.dropout_add_ln_bwd(gy, gz, z, gamma, mean, rstd, p, rng, True)
    back_old = ops.dropout_add_ln_bwd(gy, gz, z, off, mean, rstd, p, rng, True)

    zd = z.double()
    m = zd.mean(-1, keepdim=True)
    rs = torch.rsqrt((zd - m).square().mean(-1, keepdim=True) + 1e-5)
    xh = (zd - m) * rs
    g = gy.double() * gamma.double()
    dz = rs * (g - g.mean(-1, keepdim=True) - xh * (g * xh).mean(-1, keepdim=True)) + gz.double()
    ones = torch.ones_like(x)
    keep = ops.dropout_add_ln_fwd(ones, None, torch.zeros_like(x), off, None, p, 1e-5, rng)[1] != 0
    dx = dz * keep / (1 - NF.effective_dropout_p(p))
    want = [xh * gamma.double() + beta.double(), dx, dz,
            (gy.double() * xh).sum(0), gy.double().sum(0), dx.sum(0)]
    for a, b, w in zip((y, *back), (old[0], *back_old), want):
        a, b = a.double(), b.double()
        # both round once to 16 bits what differs by a few units of 2^-24 in between: no larger an error ...
        assert _error(a, w) <= 1.01 * _error(b, w) + 2e-7 * float(w.norm())
        # ... and no value further apart than neighbours in 16 bits
        step = torch.finfo(dtype).eps
        assert float(((a - b).abs() - step * torch.maximum(a.abs(), b.abs())).max()) <= 2e-5
    torch.testing.assert_close(mean, m[:, 0].float(), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(rstd, rs[:, 0].float(), rtol=1e-5, atol=0.0)


@pytest.mark.parametrize("rows,cols", [(5, 1024), (6001, 768), (300, 2560)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_alone(rows, cols, rms):
    ops = native.ops()
    torch.manual_seed(rows)
    x, gy = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(2))
    gamma, beta = (torch.randn(cols, device="cuda").bfloat16() for _ in range(2))
    off = _off_32(gamma)
    beta = None if rms else beta
    new, old = (ops.layer_norm_fwd(x, w, beta, 1e-5, rms) for w in (gamma, off))
    for a, b in zip(new, old):
        torch.testing.assert_close(a, b, rtol=2 ** -7, atol=1e-6)
    for a, b in zip(*(ops.layer_norm_bwd(gy, x, w, new[1], new[2], rms) for w in (gamma, off))):
        torch.testing.assert_close(a, b, rtol=2 ** -7, atol=2e-5)
