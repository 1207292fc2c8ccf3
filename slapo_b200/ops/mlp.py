"""Fused two-layer MLP block.

``fc_in`` is a ``LinearWithAct`` and ``fc_out`` a ``LinearWithDropout``; on CUDA the block
runs as one autograd node (:func:`slapo_b200.ops.functional.mlp`) while nothing hangs on its two
layers.  The activation given by the caller is honoured (the
reference passes it into the wrong positional slot and always gets GeLU,
slapo/op/mlp.py:39).

Parity: slapo/op/mlp.py:10-50 of the reference.
"""
from torch import nn
from torch.nn.modules import module as _module

from . import functional as NF
from .linear import LinearWithAct, LinearWithDropout


def _plain(layer, cls):
    """A layer that nothing was hung on: no hooks, collectives or replaced forward."""
    return (type(layer) is cls and layer.sync_fn is None
            and not (layer.fused_pre or layer.fused_post or layer.fused_bwd)
            and "forward" not in layer.__dict__
            and not (layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks
                     or layer._backward_pre_hooks))


def _global_hooks():
    return bool(_module._global_forward_hooks or _module._global_forward_pre_hooks
                or _module._global_backward_hooks or _module._global_backward_pre_hooks)


class FusedMLP(nn.Module):
    def __init__(self, hidden_size, intermediate_size, orig_act="gelu", resid_pdrop=0.0,
                 use_torchscript=False, device=None, dtype=None):
        super().__init__()
        self.fc_in = LinearWithAct(hidden_size, intermediate_size, bias=True, act_fn=orig_act,
                                   device=device, dtype=dtype)
        self.fc_out = LinearWithDropout(intermediate_size, hidden_size, bias=True,
                                        p=resid_pdrop, device=device, dtype=dtype)

    def forward(self, hidden_states):
        a, b = self.fc_in, self.fc_out
        if (_plain(a, LinearWithAct) and _plain(b, LinearWithDropout) and not _global_hooks()
                and NF.mlp_supported(hidden_states, a.weight, a.bias, b.weight, b.bias)):
            return NF.mlp(hidden_states, a.weight, a.bias, b.weight, b.bias, a.act_fn,
                          b.p if b.training else 0.0)
        return self.fc_out(self.fc_in(hidden_states))
