"""A linear layer with GeLU in the GEMM's epilogue: the numbers of the layer followed by bias + activation,
to the bit, in both directions; and a training step through such layers, parameter by parameter."""
import copy

import pytest
import torch

import slapo_b200 as slapo
from slapo_b200.models import BertConfig, BertForMaskedLM, mlm_loss
from slapo_b200.ops import functional as NF
from slapo_b200.ops import native

pytestmark = pytest.mark.gpu

BF, FP = torch.bfloat16, torch.float16


# few rows, steps of K in runs and one by one; every tile: one CTA of 64 / 128 / 256 columns, pairs of
# 128 / 256; ragged rows and columns
@pytest.mark.parametrize("act,dtype", [("gelu", BF), ("gelu_new", FP)])
@pytest.mark.parametrize("m,k,n", [(8, 64, 64), (16, 2048, 200), (8, 776, 3072), (40, 72, 200),
                                   (200, 768, 3072), (128, 64, 64 * 148 + 8), (120, 64, 19200),
                                   (392, 64, 4104), (2056, 64, 2056)])
def test_equals_layer_then_activation(m, k, n, act, dtype):
    torch.manual_seed(m + n)
    x = torch.randn(m, k, device="cuda", dtype=dtype, requires_grad=True)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype).requires_grad_()
    b = torch.randn(n, device="cuda", dtype=dtype, requires_grad=True)
    dy = torch.randn(m, n, device="cuda", dtype=dtype)

    def both(y):
        return [y.detach(), *torch.autograd.grad(y, [x, w, b], dy)]

    one = both(NF.linear(x, w, b, act))
    two = both(NF.bias_act(NF.linear(x, w), b, act))
    for name, p, q in zip(("y", "dx", "dw", "db"), one, two):
        assert torch.equal(p, q), name
    with torch.no_grad():
        assert torch.equal(NF.linear(x, w, b, act), one[0])
        summed = native.ops().gemm_act_fwd(x, w, b, NF._act_code(act), True, True)
        assert torch.equal(summed[0], one[0])
        assert torch.equal(summed[1], (NF.linear(x, w).float() + b.float()).to(dtype))
    # W as [in, out]: product and activation apart
    wt = w.detach().t().contiguous().requires_grad_()
    y = native.ops().linear(x, wt, b, NF._act_code(act), True)
    z = NF.linear_t(x, wt)
    assert torch.equal(y, NF.bias_act(z, b, act))
    two = torch.autograd.grad(NF.bias_act(z, b, act), [x, wt, b], dy)
    for p, q in zip(torch.autograd.grad(y, [x, wt, b], dy), two):
        assert torch.equal(p, q)
    assert native.ops().device_status() == 0


def test_gradients_of_a_step():
    """Two layers, one of them checkpointed, against the same model in 64 bits."""
    cfg = BertConfig(vocab_size=1024, hidden_size=256, num_hidden_layers=2, num_attention_heads=4,
                     intermediate_size=1024, hidden_dropout_prob=0.0, attention_probs_dropout_prob=0.0)
    torch.manual_seed(1)
    with slapo.init_empty_weights():
        model = BertForMaskedLM(cfg)
    sch = slapo.model_schedule.apply_schedule(model, "bert", model_config=cfg, bf16=True, ckpt_ratio=0.5)
    engine, _ = slapo.build(sch, target="native", config={"lr": 1e-3})
    engine.model.train()
    exact = copy.deepcopy(engine.model).double()         # plain PyTorch: no kernel takes 64 bits
    exact.zero_grad(set_to_none=True)
    ids = torch.randint(0, cfg.vocab_size, (8, 128), device="cuda")
    labels = ids.masked_fill(torch.rand(ids.shape, device="cuda") >= 0.15, -100)
    engine.backward(mlm_loss(engine(ids)["logits"], labels))
    mlm_loss(exact(ids)["logits"], labels).backward()
    want = {n: p.grad for n, p in exact.named_parameters()}
    # A gradient has come through some 15 roundings of 2^-9 per layer and direction and as many again in
    # embedding, head and loss, 90 in all, which add up like a random walk; doubled for those that
    # cancel in a parameter's sum over the tokens.
    bound = 2 * 90 ** 0.5 * 2.0 ** -9
    seen = 0
    for name, p in engine.model.named_parameters():
        err = ((p.grad.double() - want[name]).norm() / want[name].norm()).item()
        assert err < bound, (name, err)
        seen += 1
    assert seen > 30
