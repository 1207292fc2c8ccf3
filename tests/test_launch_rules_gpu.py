"""Which kernel a call gets on either side of the lines that the dispatch rules draw, from a profile of the
launch, and that both sides of a line agree with 64 bits.  The lines follow from times beside each rule."""
import math
import re

import pytest
import torch
import torch.nn.functional as F
from torch.profiler import ProfilerActivity, profile

from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16


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


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


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


# ----------------------------------------------------------- backward of the norms
def _norm_lines():
    s = sms()
    return [(4095, 512, 0.1, True, False), (4096, 512, 0.0, False, True),
            (5999, 1024, 0.1, False, False), (6000, 1024, 0.1, False, True),
            (8191, 528, 0.0, True, False), (8192, 528, 0.0, True, True),
            (8191, 768, 0.0, False, False), (8192, 1024, 0.0, False, True),
            (2 * s, 1536, 0.0, False, True), (2 * s + 1, 1536, 0.1, True, False),
            (4 * s, 1040, 0.0, False, False), (4 * s + 1, 1040, 0.1, False, True),
            (999, 2064, 0.1, True, False), (1000, 2064, 0.0, False, True)]


@pytest.mark.parametrize("line", range(14))
def test_norm_backward_lines(line):
    rows, cols, p, two, by_rows = _norm_lines()[line]
    ops = native.ops()
    torch.manual_seed(rows + cols)
    z, gy, gz = (torch.randn(rows, cols, device="cuda", dtype=FP) for _ in range(3))
    gamma = torch.randn(cols, device="cuda", dtype=FP)
    m = z.double().mean(-1, keepdim=True)
    rs = torch.rsqrt((z.double() - m).square().mean(-1, keepdim=True) + 1e-5)
    rng = torch.tensor([3, 8, 0, 0], dtype=torch.int64) if p else None
    stats = m[:, 0].float(), rs[:, 0].float()
    call = lambda: ops.dropout_add_ln_bwd(gy, gz if two else None, z, gamma, *stats, p, rng, True)
    assert of(call, "ln_bwd_rows_kernel" if by_rows else "ln_bwd_kernel")
    dx, dres, dgamma, dbeta, dbias = call()
    xh = (z.double() - m) * rs
    g = gy.double() * gamma.double()
    dz = rs * (g - g.mean(-1, keepdim=True) - xh * (g * xh).mean(-1, keepdim=True))
    if two:
        dz = dz + gz.double()
    close(dres, dz, FP)
    close(dgamma, (gy.double() * xh).sum(0), FP)
    close(dbeta, gy.double().sum(0), FP)
    keep = dx != 0 if p else torch.ones_like(dx, dtype=torch.bool)
    from slapo_b200.ops import functional as NF
    want = dz * keep / (1 - (NF.effective_dropout_p(p) if p else 0.0))
    close(dx, want, FP)
    close(dbias, want.sum(0), FP)


# ----------------------------------------------------------- forward of attention, short calls
def _attn_lines():
    s = sms()
    # heads, queries, keys, head dim, causal, dropout, key bias; softmax groups or not
    # (two row tiles for 129 - 256 queries)
    return [(s, 200, 100, 64, False, 0.0, False, False),
            (s + 1, 200, 100, 64, False, 0.0, False, True),
            (s, 256, 128, 32, False, 0.1, True, False),
            (8, 130, 64, 64, False, 0.0, False, False),
            (s // 2, 200, 256, 64, False, 0.0, False, True),
            (s // 2 + 1, 200, 256, 64, False, 0.0, False, False),
            (s // 2 + 1, 200, 256, 64, False, 0.1, False, True),
            (s // 2 + 1, 200, 256, 64, False, 0.1, True, False),
            (s // 2 + 1, 200, 200, 64, True, 0.1, False, False),
            (s - 20, 200, 300, 64, False, 0.0, True, False),
            (s - 20, 200, 400, 64, False, 0.0, True, True),
            (s - 20, 200, 100, 128, False, 0.0, False, True),
            (s - 20, 100, 100, 64, False, 0.0, False, False)]


@pytest.mark.parametrize("line", range(13))
def test_attention_forward_lines(line):
    h, sq, sk, d, causal, p, biased, groups = _attn_lines()[line]
    ops = native.ops()
    torch.manual_seed(h + sq)
    q, k, v = (torch.randn(1, s, h, d, device="cuda", dtype=BF) for s in (sq, sk, sk))
    kb = torch.randn(1, sk, device="cuda") if biased else None
    rng = torch.tensor([3, 8, 0, 0], dtype=torch.int64) if p else None
    call = lambda: ops.flash_attn_fwd(q, k, v, kb, None, causal, d ** -0.5, p, rng)
    assert of(call, "flash_fwd_groups_kernel" if groups else "flash_fwd_kernel")
    out, lse = call()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * d ** -0.5
    if biased:
        s = s + kb.double()[:, None, None]
    if causal:
        s = s.masked_fill(torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1), -math.inf)
    torch.testing.assert_close(lse.double(), torch.logsumexp(s, -1).view_as(lse), rtol=1e-5, atol=2e-5)
    if not p:      # (dropped calls: tests/test_flash_paths_gpu.py)
        close(out, torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double()), BF, roundings=2)
    assert ops.device_status() == 0
