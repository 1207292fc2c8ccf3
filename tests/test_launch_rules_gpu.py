"""Which kernel a call gets on either side of the lines that the dispatch rules draw, from a profile of the
launch, and that both sides of a line agree with 64 bits.  The lines follow from times beside each rule."""
import re

import pytest
import torch
import torch.nn.functional as F
from torch.profiler import ProfilerActivity, profile

from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def launched(call):
    """Names of the kernels that ``call`` launches, without their namespace and arguments."""
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as seen:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in seen.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    ours = (re.search(r"slapo::(\w+(?:<[^(]*>)?)\(", n) for n in names)
    return [m.group(1) for m in ours if m]


def of(call, what):
    """The name, with its template arguments, of the one kernel of ``call`` that starts with ``what``."""
    names = launched(call)
    if not names:
        pytest.skip("no profile of kernels on this machine")
    (name,) = [n for n in names if n.startswith(what)]
    return name


def close(got, want, dtype, roundings=1):
    """Each rounding to 16 bits is up to 2^-9 (bf16) or 2^-12 (fp16) relative; four times that."""
    err = ((got.double() - want).norm() / want.norm()).item()
    assert err < roundings * 4 * 2.0 ** (-9 if dtype == BF else -12), err


# ----------------------------------------------------------- epilogue warps of the CTA-pair product
@pytest.mark.parametrize("m,n,k,b_mn,warps", [
    (8192, 4096, 1024, False, 16), (8192, 4096, 1032, False, 8), (8192, 4096, 512, True, 8),
    (19 * 256, 2048, 512, False, 16),          # 152 tiles: more than two rounds of 74 pairs
    (18 * 256, 2048, 512, False, 8), (1000, 2048, 512, False, 8)])
def test_epilogue_warps_of_plain_products(m, n, k, b_mn, warps):
    ops = native.ops()
    torch.manual_seed(m + k)
    a = torch.randn(m, k, device="cuda", dtype=BF)
    b = (torch.randn(*((k, n) if b_mn else (n, k)), device="cuda") * k ** -0.5).to(BF)
    bias = torch.randn(n, device="cuda", dtype=BF)
    assert of(lambda: ops.gemm(a, b, bias, -1, False, b_mn), "gemm2_tc05").endswith(f", {warps}>")
    want = a.double() @ (b if b_mn else b.t()).double() + bias.double()
    close(ops.gemm(a, b, bias, -1, False, b_mn), want, BF)


@pytest.mark.parametrize("m,n,k", [(4096, 4096, 512), (2056, 2056, 72), (1000, 2048, 512)])
def test_epilogue_warps_of_activations(m, n, k):
    ops = native.ops()
    wide = tuple(ops.gemm_tile(m, n)) == (True, 0)
    assert wide or tuple(ops.gemm_tile(m, n)) == (True, 128)
    torch.manual_seed(m)
    x, z = torch.randn(m, k, device="cuda", dtype=BF), torch.randn(m, n, device="cuda", dtype=BF)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(BF)
    w2 = w.t().contiguous()
    b = torch.randn(n, device="cuda", dtype=BF)
    pre = F.linear(x.double(), w.double(), b.double())
    for act in (0, 1):
        want = F.gelu(pre, approximate="tanh" if act else "none")
        for keep in (False, True):
            call = lambda: ops.gemm_act_fwd(x, w, b, act, keep, True)
            many = wide and not (act == 1 and keep)
            assert of(call, "gemm2_tc05").endswith(f", {16 if many else 8}>")
            close(call()[0], want, BF, roundings=2)
    for act in (0, 1, 2):
        call = lambda: ops.gemm_act_bwd(x, w2, z, act)
        assert of(call, "gemm2_tc05").endswith(f", {16 if wide and act == 0 else 8}>")
    if n % 16 == 0:
        rng = torch.tensor([5, 4, 0, 0], dtype=torch.int64)
        call = lambda: ops.gemm_dropout_fwd(x, w, b, 0.1, rng)
        assert of(call, "gemm2_tc05").endswith(f", {16 if wide else 8}>")
        plain = ops.bias_dropout_add_fwd(ops.gemm(x, w, None, -1, False, False), b, None, 0.1, rng)
        assert torch.equal(call(), plain)
