"""Host side of the fused tensor-parallel linears: forward and backward of each layer function on
the CPU, for a group of one rank, with the GEMM operators and the collective kernels restated in
PyTorch (a name or an argument that no longer fits fails here, without a GPU)."""
import types

import pytest
import torch
import torch.nn.functional as F

from slapo_b200.ops import functional as NF
from slapo_b200.parallel import fused_tp as ft


def _gemm(a, b, bias=None, act=-1, a_mn=False, b_mn=False, out=None, pre_act=None, split_k=False):
    y = (a.t() if a_mn else a) @ (b if b_mn else b.t())
    return y if bias is None else y + bias


def _gemm_out(a, b, bias, act, a_mn, b_mn, out, pre_act, impl, split_k):
    return _gemm(a, b, bias, act, a_mn, b_mn)


@pytest.fixture
def one_rank(monkeypatch):
    ops = types.SimpleNamespace(gemm_out=_gemm_out, colsum=lambda t: t.sum(0))
    monkeypatch.setattr(NF.native, "ops", lambda: ops)
    monkeypatch.setattr(NF, "gemm_supported", lambda x, w: True)

    def product(ctx, x, w, bias=None, b_mn=False, **kw):
        return _gemm(x, w, bias, b_mn=b_mn)

    monkeypatch.setattr(ft, "gemm_ar", product)
    monkeypatch.setattr(ft, "gemm_rs", product)
    monkeypatch.setattr(ft, "ag_gemm", lambda ctx, x, w, bias=None, b_mn=False, **kw:
                        (_gemm(x, w, bias, b_mn=b_mn), x))
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda t, group=None: None)
    return types.SimpleNamespace(world=1, rank=0, nvls=False, group=None)


@pytest.mark.parametrize("fn", ["col_linear_ar_bwd", "ag_linear", "rs_linear", "ar_linear"])
@pytest.mark.parametrize("has_bias", [True, False])
@pytest.mark.parametrize("layout", ["dense", "strided", "columns"])
def test_layer_functions(one_rank, fn, has_bias, layout):
    torch.manual_seed(0)
    t, b, k, n = 128, 2, 16, 24       # 256 rows: whole blocks of the fused input gradient
    if layout == "strided":
        x = torch.randn(t, b, 3 * k)[..., k:2 * k]
    elif layout == "columns":
        x = torch.randn(k, b, t).permute(2, 1, 0)
    else:
        x = torch.randn(t, b, k)
    x = x.detach().requires_grad_()
    w = torch.randn(n, k, requires_grad=True)
    bias = torch.randn(n, requires_grad=True) if has_bias else None
    leaves = [p for p in (x, w, bias) if p is not None]
    y = getattr(ft, fn)(x, w, bias, one_rank)
    dy = torch.randn_like(y)
    want = F.linear(x, w, bias)
    torch.testing.assert_close(y, want)
    for got, ref in zip(torch.autograd.grad(y, leaves, dy), torch.autograd.grad(want, leaves, dy)):
        torch.testing.assert_close(got, ref, rtol=1e-4, atol=1e-4)


def test_rows_of_an_odd_batch(one_rank):
    """Row counts that do not divide into the fused kernel's blocks all-reduce after the GEMM."""
    x = torch.randn(5, 16, requires_grad=True)
    w = torch.randn(24, 16, requires_grad=True)
    y = ft.col_linear_ar_bwd(x, w, None, one_rank)
    y.sum().backward()
    torch.testing.assert_close(x.grad, w.detach().sum(0).expand(5, 16))
