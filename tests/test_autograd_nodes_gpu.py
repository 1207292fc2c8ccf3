"""What autograd asks of the layers' nodes beside the gradients themselves: graphs that are freed or
kept, saved-tensor hooks, inputs that need no gradient, modes that have no rule."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _leaf(*shape):
    return torch.randn(*shape, device="cuda", dtype=BF).requires_grad_()


def _layers():
    """name -> (function of the leaves, leaves)"""
    h = 64
    attn = (_leaf(2, 40, 2, h), _leaf(2, 40, 2, h), _leaf(2, 40, 2, h))
    return {
        "linear": (lambda x, w, b: NF.linear(x, w, b), (_leaf(24, h), _leaf(48, h), _leaf(48))),
        "linear_relu": (lambda x, w, b: NF.linear(x, w, b, "relu"),
                        (_leaf(24, h), _leaf(48, h), _leaf(48))),
        "linear_gelu": (lambda x, w, b: NF.linear(x, w, b, "gelu"),
                        (_leaf(24, h), _leaf(48, h), _leaf(48))),
        "linear_t": (lambda x, w, b: NF.linear_t(x, w, b), (_leaf(24, h), _leaf(h, 48), _leaf(48))),
        "bias_act": (lambda x, b: NF.bias_act(x, b, "gelu"), (_leaf(24, h), _leaf(h))),
        "layer_norm": (lambda x, w, b: NF.layer_norm(x, w, b), (_leaf(24, h), _leaf(h), _leaf(h))),
        "rms_norm": (lambda x, w: NF.rms_norm(x, w), (_leaf(24, h), _leaf(h))),
        "dropout_add_norm": (lambda x, b, r, w, lb: NF.dropout_add_layer_norm(
            x, b, r, w, lb, 0.0, 1e-5)[0], (_leaf(24, h), _leaf(h), _leaf(24, h), _leaf(h), _leaf(h))),
        "attention": (lambda q, k, v: NF.flash_attention(q, k, v, causal=True), attn),
    }


NAMES = list(_layers()) if torch.cuda.is_available() else [
    "linear", "linear_relu", "linear_gelu", "linear_t", "bias_act", "layer_norm", "rms_norm",
    "dropout_add_norm", "attention"]


@pytest.mark.parametrize("name", NAMES)
def test_graph_freed_or_kept(name):
    fn, leaves = _layers()[name]
    y = fn(*leaves)
    dy = torch.randn_like(y)
    first = torch.autograd.grad(y, leaves, dy, retain_graph=True)
    second = torch.autograd.grad(y, leaves, dy)
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y, leaves, dy)


@pytest.mark.parametrize("name", NAMES)
def test_saved_tensor_hooks(name):
    """Offloading what a node saves changes nothing, and every node saves through the hooks."""
    fn, leaves = _layers()[name]
    y = fn(*leaves)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy)
    packed = []

    def pack(t):
        packed.append(t.shape)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = fn(*leaves)
    assert packed
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, leaves, dy), want))


@pytest.mark.parametrize("name", NAMES)
def test_each_input_alone(name):
    fn, leaves = _layers()[name]
    y = fn(*leaves)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy)
    for i, leaf in enumerate(leaves):
        y = fn(*(t if j == i else t.detach() for j, t in enumerate(leaves)))
        (got,) = torch.autograd.grad(y, leaf, dy)
        assert torch.equal(got, want[i]), i
    assert not fn(*(t.detach() for t in leaves)).requires_grad


@pytest.mark.parametrize("name", NAMES)
def test_modes_without_a_rule_are_refused(name):
    fn, leaves = _layers()[name]
    plain = [t.detach() for t in leaves]
    with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        fn(fwd.make_dual(plain[0], torch.ones_like(plain[0])), *leaves[1:])
    with pytest.raises(RuntimeError):
        torch.vmap(lambda t: fn(t, *plain[1:]))(torch.stack([plain[0], plain[0]]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: fn(t, *plain[1:]).float().sum())(plain[0])
    with pytest.raises(RuntimeError):
        torch.vmap(lambda t: NF.bias_dropout_add(t, None, None, 0.5))(torch.randn(2, 8, 64, device="cuda"))
    assert native.ops().device_status() == 0


def test_a_refusal_in_the_backward_thread_is_an_error():
    """Weight gradients contract over the tokens, which the GEMM takes in eights."""
    w = _leaf(48, 64)
    y = NF.linear(torch.randn(12, 64, device="cuda", dtype=BF), w)
    with pytest.raises(RuntimeError, match="gemm: launch refused"):
        y.sum().backward()
