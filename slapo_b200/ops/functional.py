"""Functional front ends of the fused element-wise / normalisation ops.

Every function has two implementations with identical semantics:

* CUDA tensors run the hand-written sm_100a kernels of the ``_C`` extension
  (one pass over HBM for the forward, one for the backward, dropout masks
  regenerated from a Philox ``(seed, offset)`` pair instead of being stored);
* anything else (CPU tensors, meta tensors, fx proxies) runs plain PyTorch,
  which is also the numerical oracle of the kernel tests.

A CUDA tensor with the extension missing is an error unless the environment
variable ``SLAPO_B200_ALLOW_FALLBACK=1`` is set: a silent eager fallback on a
GPU would hide a broken build.
"""
from __future__ import annotations

import math
import os

import torch
import torch.nn.functional as F

from . import native

_TANH_ACTS = ("gelu_new", "gelu_tanh", "gelu_pytorch_tanh")


def _native_ok(*tensors) -> bool:
    t = next((x for x in tensors if torch.is_tensor(x)), None)
    if t is None or not isinstance(t, torch.Tensor) or not t.is_cuda:
        return False
    if t.dtype not in (torch.bfloat16, torch.float16, torch.float32):
        return False
    if native.available():
        return True
    if os.environ.get("SLAPO_B200_ALLOW_FALLBACK", "0") == "1":
        return False
    raise RuntimeError(
        "slapo_b200 native extension is not built/loaded but a CUDA tensor was given; "
        "run `python -c 'import __graft_entry__ as g; g.build()'` or set "
        "SLAPO_B200_ALLOW_FALLBACK=1 to accept the eager PyTorch path")


def _nodes():
    """The extension's operators, for those with an autograd node of their own.  functorch has no
    rule for such a node: vmap would run it slice by slice, whatever its ``randomness`` says."""
    if torch._C._functorch.peek_interpreter_stack() is not None:
        raise RuntimeError("slapo_b200's CUDA layers do not support functorch transforms "
                           "(vmap, grad, jvp, ...)")
    return native.ops()


# ---------------------------------------------------------------------- #
# activations
def _act_ref(x, act):
    if act == "gelu":
        return F.gelu(x)
    if act in _TANH_ACTS:
        return F.gelu(x, approximate="tanh")
    if act == "relu":
        return F.relu(x)
    raise NotImplementedError(act)


def _act_code(act):
    return {"gelu": 0, "relu": 2}.get(act, 1)


def bias_act(x, bias, act: str = "gelu"):
    """``act(x + bias)``; act in gelu (erf) / gelu_new (tanh) / relu."""
    if _native_ok(x) and x.shape[-1] % 8 == 0:
        return _nodes().bias_act(x, bias, _act_code(act))
    return _act_ref(x + bias if bias is not None else x, act)


def bias_gelu(x, bias, approximate: str = "none"):
    return bias_act(x, bias, "gelu" if approximate == "none" else "gelu_new")


# ---------------------------------------------------------------------- #
# linear layers on the tcgen05 GEMM
def gemm_supported(x, weight) -> bool:
    """CUDA 16-bit operands whose dimensions TMA can address (multiples of 8 elements)."""
    if not (torch.is_tensor(x) and x.is_cuda and x.dtype in (torch.bfloat16, torch.float16)):
        return False
    if weight.dtype != x.dtype or weight.dim() != 2 or weight.stride(1) != 1:
        return False
    if os.environ.get("SLAPO_B200_LIBRARY_GEMM", "0") == "1":   # A/B switch for measurements
        return False
    return (x.shape[-1] % 8 == 0 and weight.shape[0] % 8 == 0 and weight.stride(0) % 8 == 0
            and x.numel() > 0 and _native_ok(x))


def gemm(a, b, bias=None, act=-1, a_mn=False, b_mn=False, out=None, pre_act=None, split_k=False):
    """``act(A B^T + bias)`` on this library's tcgen05 kernels (CTA pairs where the problem
    has a pair tile).  ``a_mn`` / ``b_mn``: the operand is stored ``[K, M]`` / ``[K, N]``."""
    return native.ops().gemm_out(a, b, bias, act, a_mn, b_mn, out, pre_act, 0, split_k)


_RELU = 2


def linear_t(x, weight, bias=None):
    """``x @ weight + bias`` for a weight stored ``[in_features, out_features]``."""
    if (torch.is_tensor(x) and x.is_cuda and x.dtype in (torch.bfloat16, torch.float16)
            and weight.dtype == x.dtype and weight.dim() == 2 and weight.stride(1) == 1
            and weight.shape[0] % 8 == 0 and weight.shape[1] % 8 == 0 and weight.stride(0) % 8 == 0
            and x.numel() > 0 and os.environ.get("SLAPO_B200_LIBRARY_GEMM", "0") != "1"
            and _native_ok(x)):
        return _nodes().linear(x, weight, bias, -1, True)
    out = torch.matmul(x, weight)
    return out if bias is None else out + bias


def linear(x, weight, bias=None, act=None):
    """``act(x @ weight.T + bias)``; ``act`` in None / "gelu" / "gelu_new" / "relu".  CUDA
    16-bit tensors run this library's GEMM (bias and activation in its epilogue), anything
    else PyTorch."""
    if gemm_supported(x, weight):
        nodes = _nodes()
        if act is None or act == "relu":
            return nodes.linear(x, weight, bias, -1 if act is None else _RELU, False)
        if _epilogue_bias(bias, x):
            return nodes.linear(x, weight, bias, _act_code(act), False)
        return bias_act(nodes.linear(x, weight, None, -1, False), bias, act)
    out = F.linear(x, weight, bias)
    return out if act is None else _act_ref(out, act)


def _epilogue_bias(bias, x):
    """Whether a GEMM's epilogue can add ``bias`` in 16-byte words."""
    return (bias is not None and bias.dtype == x.dtype and bias.is_contiguous()
            and bias.data_ptr() % 16 == 0)


def mlp_supported(x, w1, b1, w2, b2) -> bool:
    """Whether :func:`mlp` takes a feed-forward block: what its two GEMMs take."""
    if not gemm_supported(x, w1):
        return False
    _nodes()        # (a transform is refused before the biases' addresses are looked at)
    return (w2.dtype == x.dtype and w2.dim() == 2 and w2.stride(1) == 1
            and w2.shape[0] % 8 == 0 and w2.stride(0) % 8 == 0 and w1.shape[1] == x.shape[-1]
            and w2.shape[1] == w1.shape[0] and _epilogue_bias(b1, x) and _epilogue_bias(b2, x))


def mlp(x, w1, b1, w2, b2, act: str, p: float):
    """``dropout(act(x @ w1.T + b1) @ w2.T + b2, p)`` as one autograd node."""
    return _nodes().mlp(x, w1, b1, w2, b2, _act_code(act), p)


# ---------------------------------------------------------------------- #
# dropout family
def effective_dropout_p(p: float) -> float:
    """Dropout probability the CUDA kernels actually apply.  They draw 7-bit
    random numbers (16 decisions per Philox call), so ``p`` is rounded to a
    multiple of 1/128 (0.1 -> 13/128 = 0.1016); kept values are rescaled by
    ``1 / (1 - effective p)``, which keeps the expectation exact."""
    return min(max(int(p * 128.0 + 0.5), 0), 127) / 128.0


def bias_dropout_add(x, bias, residual, p: float, training: bool = True):
    """``dropout(x + bias, p) + residual`` (bias / residual may be None)."""
    if _native_ok(x) and training and p > 0.0 and x.shape[-1] % 8 == 0:
        return _nodes().bias_dropout_add(x, bias, residual, p)
    out = x + bias if bias is not None else x
    out = F.dropout(out, p, training)
    return out + residual if residual is not None else out


def bias_dropout(x, bias, p: float, training: bool = True):
    return bias_dropout_add(x, bias, None, p, training)


# ---------------------------------------------------------------------- #
# normalisation
def layer_norm(x, weight, bias, eps: float = 1e-5):
    if _native_ok(x) and x.shape[-1] % 8 == 0 and x.shape[-1] <= 16384:
        return _nodes().norm(x, weight, bias, eps, False)
    return F.layer_norm(x, (x.shape[-1],), weight, bias, eps)


def rms_norm(x, weight, eps: float = 1e-6):
    """T5-style RMS norm: no mean subtraction, no bias, fp32 statistics."""
    if _native_ok(x) and x.shape[-1] % 8 == 0 and x.shape[-1] <= 16384:
        return _nodes().norm(x, weight, None, eps, True)
    var = x.float().pow(2).mean(-1, keepdim=True)
    return (x.float() * torch.rsqrt(var + eps)).to(x.dtype) * weight


def dropout_add_layer_norm(x, bias, residual, weight, ln_bias, p: float, eps: float,
                           training: bool = True):
    """``z = dropout(x + bias) + residual; y = LayerNorm(z)``; returns ``(y, z)``.

    ``z`` is returned because a pre-LN block needs it as the next residual; a
    post-LN block (BERT) just drops it."""
    if _native_ok(x) and x.shape[-1] % 8 == 0 and x.shape[-1] <= 16384:
        return _nodes().dropout_add_norm(x, bias, residual, weight, ln_bias,
                                         p if training else 0.0, eps)
    z = x + bias if bias is not None else x
    z = F.dropout(z, p, training) + residual
    return F.layer_norm(z, (z.shape[-1],), weight, ln_bias, eps), z


# ---------------------------------------------------------------------- #
# attention
def t5_relative_position_bucket(relative_position, bidirectional=True, num_buckets=32,
                                max_distance=128):
    """T5 bucket index of ``relative_position = key_pos - query_pos``."""
    ret = torch.zeros_like(relative_position)
    n = num_buckets
    if bidirectional:
        n //= 2
        ret = ret + (relative_position > 0).to(torch.long) * n
        rp = relative_position.abs()
    else:
        rp = -torch.min(relative_position, torch.zeros_like(relative_position))
    max_exact = n // 2
    is_small = rp < max_exact
    large = max_exact + (
        torch.log(rp.float().clamp(min=1) / max_exact) / math.log(max_distance / max_exact)
        * (n - max_exact)).to(torch.long)
    large = torch.min(large, torch.full_like(large, n - 1))
    return ret + torch.where(is_small, rp, large)


def attention_reference(q, k, v, key_padding_bias=None, causal=False, scale=None,
                        dropout_p=0.0, training=False, rel_bias_table=None,
                        rel_bidirectional=True, rel_max_distance=128, dropout_mask=None,
                        attn_bias=None):
    """Plain-PyTorch attention on ``[B, S, H, D]`` tensors (the oracle).

    ``key_padding_bias`` is an additive ``[B, Sk]`` bias (0 / large negative);
    ``rel_bias_table`` a ``[num_buckets, H]`` T5 relative-position table; ``attn_bias`` any
    additive bias that broadcasts to ``[B, H, Sq, Sk]`` (only this function takes one)."""
    b, sq, h, d = q.shape
    sk = k.shape[1]
    scale = (1.0 / math.sqrt(d)) if scale is None else scale
    qf, kf, vf = (t.transpose(1, 2).float() for t in (q, k, v))
    scores = torch.matmul(qf, kf.transpose(-1, -2)) * scale
    if rel_bias_table is not None:
        ctx_pos = torch.arange(sq, device=q.device)[:, None] + (sk - sq)
        mem_pos = torch.arange(sk, device=q.device)[None, :]
        buckets = t5_relative_position_bucket(
            mem_pos - ctx_pos, rel_bidirectional, rel_bias_table.shape[0], rel_max_distance)
        scores = scores + rel_bias_table.float()[buckets].permute(2, 0, 1)[None]
    if key_padding_bias is not None:
        scores = scores + key_padding_bias.float().view(b, 1, 1, sk)
    if attn_bias is not None:
        scores = scores + attn_bias.float()
    if causal:
        keep = torch.ones(sq, sk, dtype=torch.bool, device=q.device).tril(diagonal=sk - sq)
        scores = scores.masked_fill(~keep, float("-inf"))
    probs = torch.softmax(scores, dim=-1)
    if dropout_mask is not None:
        probs = probs * dropout_mask / (1.0 - dropout_p)
    elif dropout_p > 0.0 and training:
        probs = F.dropout(probs, dropout_p, True)
    out = torch.matmul(probs, vf)
    return out.transpose(1, 2).to(q.dtype)


def _transformed(tensors):
    """Whether a functorch transform or forward-mode differentiation is at work on them."""
    return torch.autograd.forward_ad._current_level >= 0 or any(
        torch._C._functorch.is_functorch_wrapped_tensor(t) for t in tensors)


def append_kv(past_k, past_v, k, v):
    """Key / value caches ``[B, S, H, D]`` followed by the new tokens ``[B, n, H, D]``: two new
    tensors.  ``k`` and ``v`` may be slices of a packed projection output, read in place by one
    kernel; the operator concatenates what that does not take."""
    if (type(k) is torch.Tensor and _native_ok(k)
            and torch._C._functorch.peek_interpreter_stack() is None):
        return native.ops().append_kv(past_k, past_v, k, v)
    return torch.cat((past_k, k), dim=1), torch.cat((past_v, v), dim=1)


_FALLBACK_SEEN = set()


def _warn_attention_fallback(q, k):
    """One WARNING per (dtype, head dim, layout problem): a CUDA attention call that the
    tcgen05 kernels do not take runs the fp32 reference with a materialised [B, H, Sq, Sk]
    score matrix - correct, but many times slower and memory-hungry."""
    why = []
    if q.dtype not in (torch.bfloat16, torch.float16):
        why.append(f"dtype {q.dtype} (kernels: bf16 / fp16)")
    d = q.shape[-1]
    if not (8 <= d <= 128 and d % 8 == 0):
        why.append(f"head dim {d} (kernels: multiples of 8 up to 128)")
    if q.dim() != 4:
        why.append(f"{q.dim()}-D input (kernels: [B, S, H, D])")
    if not why:
        why.append("strides or alignment (D contiguous, other strides multiples of 8 "
                   "elements, 16-byte aligned data)")
    key = (q.dtype, d, tuple(why))
    if key in _FALLBACK_SEEN:
        return
    _FALLBACK_SEEN.add(key)
    import logging

    logging.getLogger("slapo_b200.ops").warning(
        "flash_attention falls back to the PyTorch reference for q %s / k %s: %s",
        tuple(q.shape), tuple(k.shape), "; ".join(why))


def flash_attention(q, k, v, key_padding_bias=None, causal=False, scale=None, dropout_p=0.0,
                    training=True, rel_bias_table=None, rel_bidirectional=True,
                    rel_max_distance=128):
    """Attention on ``[B, S, H, D]`` tensors (any strides on B/S/H, D
    contiguous).  CUDA bf16/fp16 inputs run the tcgen05 flash kernels."""
    from .flash_attn import flash_attention_native, native_supported

    if torch.is_tensor(q) and q.is_cuda and native_supported(q, k, v):
        _native_ok(q)
        return flash_attention_native(q, k, v, key_padding_bias, causal, scale,
                                      dropout_p if training else 0.0, rel_bias_table,
                                      rel_bidirectional, rel_max_distance)
    if torch.is_tensor(q) and q.is_cuda:
        _warn_attention_fallback(q, k)
    return attention_reference(q, k, v, key_padding_bias, causal, scale, dropout_p, training,
                               rel_bias_table, rel_bidirectional, rel_max_distance)
