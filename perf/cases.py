"""The work that users of this framework have it do, as cases that can be timed and compared.

Training steps of transformer layers carry the framework's main path: attention (packed and
separate projections, causal and not, with padding masks, dropout and T5's relative bias), the
fused MLP, the fused normalisations, the language-model loss and a whole optimizer step; generation
adds the one-token attention block over a key / value cache and inference a small forward pass.
Sizes are those of the BERT, GPT-2, GPT-Neo, OPT and T5 configurations of this repository.

``exact`` restates every layer in 64-bit PyTorch.  The dropout masks it needs are restated as
well: Philox4x32 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC'11) with seven
rounds, one call per 16 consecutive elements, 7-bit draws.
"""
import math
import re

import torch
import torch.nn.functional as F

import slapo_b200 as slapo
from slapo_b200.models import BertConfig, BertForMaskedLM, mlm_loss
from slapo_b200.op import (FlashAttention, FlashAttentionOp, FusedDropoutAddLayerNorm,
                           FusedLayerNorm, FusedMLP, FusedRMSNorm, ParallelCrossEntropy)
from slapo_b200.ops.linear import adopt_native_linears

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # BERT-large's attention as its schedule runs it in training: packed QKV, 32 x 512 tokens
        {"name": "attn_bert_large", "kind": "attn", "batch": 32, "sq": 512, "sk": 512, "heads": 16,
         "dim": 64, "packed": True, "causal": False, "mask": False, "rel": False, "p": 0.1,
         "train": True, "dtype": "bf16"},
        # GPT-Neo-1.3B's attention at its full context
        {"name": "attn_gpt_neo", "kind": "attn", "batch": 4, "sq": 2048, "sk": 2048, "heads": 16,
         "dim": 128, "packed": True, "causal": True, "mask": False, "rel": False, "p": 0.0,
         "train": True, "dtype": "bf16"},
        # OPT-2.7B's heads of 80 on right-padded prompts of an odd length
        {"name": "attn_opt_ragged", "kind": "attn", "batch": 4, "sq": 1000, "sk": 1000,
         "heads": 32, "dim": 80, "packed": False, "causal": True, "mask": True, "rel": False,
         "p": 0.0, "train": True, "dtype": "fp16"},
        # the first layer of a T5-large encoder: relative-position table and its gradient
        {"name": "attn_t5", "kind": "attn", "batch": 8, "sq": 512, "sk": 512, "heads": 16,
         "dim": 64, "packed": False, "causal": False, "mask": True, "rel": True, "p": 0.1,
         "train": True, "dtype": "bf16"},
        # one generated token of GPT-Neo-1.3B's attention block for eight sequences
        {"name": "block_decode", "kind": "decode", "batch": 8, "new": 1, "past": 1500, "heads": 16,
         "dim": 128, "dtype": "bf16"},
        # the feed-forward block of GPT-2 medium / BERT-large at the benchmark's 16384 tokens
        {"name": "mlp_large", "kind": "mlp", "tokens": 16384, "hidden": 1024, "inner": 4096,
         "act": "gelu", "p": 0.1, "dtype": "bf16"},
        # OPT-2.7B's feed-forward sizes, one micro-batch of 4 x 1024
        {"name": "mlp_opt", "kind": "mlp", "tokens": 4096, "hidden": 2560, "inner": 10240,
         "act": "relu", "p": 0.0, "dtype": "bf16"},
        # GPT-2 small on one short sequence: launches and host time count
        {"name": "mlp_small", "kind": "mlp", "tokens": 200, "hidden": 768, "inner": 3072,
         "act": "gelu_new", "p": 0.1, "dtype": "fp16"},
        # the tail of every BERT-large block in training
        {"name": "norm_bert", "kind": "norm", "form": "dropout_add", "tokens": 16384,
         "hidden": 1024, "p": 0.1, "dtype": "bf16"},
        # next-token loss over GPT-2's padded vocabulary
        {"name": "ce_lm", "kind": "ce", "tokens": 8192, "vocab": 50304, "keep": 1.0,
         "dtype": "bf16"},
        # one short sentence through a two-layer BERT-base: the smallest whole call
        {"name": "bert_infer", "kind": "infer", "layers": 2, "hidden": 768, "heads": 12,
         "inner": 3072, "vocab": 30528, "batch": 1, "seq": 128, "dtype": "bf16"},
        # a training step at BERT-large's width through the native engine, as the benchmark
        # runs it (four of its layers, every other one checkpointed)
        {"name": "bert_step", "kind": "step", "layers": 4, "hidden": 1024, "heads": 16,
         "inner": 4096, "vocab": 30528, "batch": 16, "seq": 512, "p": 0.1, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "mlp", "mlp", "norm", "ce", "decode", "infer",
                       "step"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "attn":
        dim = rng.choice([32, 64, 64, 80, 128])
        heads = rng.choice([4, 8, 12, 16, 20, 32])
        packed = rng.random() < 0.5
        sq = _log(rng, 48, 2048)
        causal = rng.random() < 0.5
        sk = sq if packed or causal or rng.random() < 0.6 else _log(rng, 48, 2048)
        most = max(1, min(16384 // max(sq, sk), int(1.7e10 / (heads * sq * sk * dim))))
        return {"kind": "attn", "batch": rng.randint(1, min(32, most)), "sq": sq, "sk": sk,
                "heads": heads, "dim": dim, "packed": packed, "causal": causal,
                "mask": rng.random() < 0.4, "rel": sq == sk and rng.random() < 0.25,
                "p": rng.choice([0.0, 0.1]), "train": rng.random() < 0.75, "dtype": half}
    if kind == "mlp":
        hidden = rng.choice([512, 768, 1024, 1536, 2048, 2560])
        # (weight gradients contract over the tokens, which the framework takes in eights)
        tokens = _log(rng, 4, 2048 * 1024 * 1024 // hidden ** 2) * 8
        return {"kind": "mlp", "tokens": tokens,
                "hidden": hidden, "inner": 4 * hidden,
                "act": rng.choice(["gelu", "gelu_new", "relu"]), "p": rng.choice([0.0, 0.1]),
                "dtype": half}
    if kind == "norm":
        hidden = rng.choice([512, 768, 1024, 2048, 2560])
        return {"kind": "norm", "form": rng.choice(["dropout_add", "layer", "rms"]),
                "tokens": _log(rng, 32, 16384 * 1024 // hidden), "hidden": hidden,
                "p": rng.choice([0.0, 0.1]), "dtype": rng.choice(["bf16", "fp16", "fp32"])}
    if kind == "ce":
        return {"kind": "ce", "tokens": _log(rng, 64, 8192),
                "vocab": rng.choice([30528, 32128, 50272, 50304]),
                "keep": rng.choice([0.15, 1.0]), "dtype": half}
    if kind == "decode":
        return {"kind": "decode", "batch": _log(rng, 1, 16), "new": rng.choice([1, 1, 1, 5]),
                "past": _log(rng, 16, 2000), "heads": rng.choice([12, 16, 20]),
                "dim": rng.choice([64, 128]), "dtype": half}
    if kind == "infer":
        return {"kind": "infer", "layers": rng.randint(1, 4), "hidden": 768, "heads": 12,
                "inner": 3072, "vocab": 30528, "batch": rng.randint(1, 8),
                "seq": _log(rng, 16, 512), "dtype": half}
    return {"kind": "step", "layers": rng.randint(1, 4), "hidden": 1024, "heads": 16,
            "inner": 4096, "vocab": 30528, "batch": rng.randint(1, 16),
            "seq": 8 * _log(rng, 8, 64), "p": rng.choice([0.0, 0.1]), "dtype": "bf16"}


# --------------------------------------------------------------------------- #
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(gen, shape, std, dtype, mean=0.0):
    return (torch.randn(shape, generator=gen, device=DEV) * std + mean).to(dtype)


def _padding(gen, batch, sk):
    """Additive mask [B, 1, 1, Sk] of right-padded sequences, at least half of each real."""
    length = torch.randint((sk + 1) // 2, sk + 1, (batch, 1), generator=gen, device=DEV)
    pad = torch.arange(sk, device=DEV)[None, :] >= length
    return (pad.float() * -10000.0)[:, None, None, :]


def _attn_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    b, sq, sk, h, d = (case[k] for k in ("batch", "sq", "sk", "heads", "dim"))
    qs = d ** -0.25 if case["rel"] else 1.0       # T5 multiplies no 1 / sqrt(d)
    if case["packed"] and not case["rel"]:
        t = {"qkv": _normal(g, (b, sq, h, 3, d), 1.0, dt)}
    else:
        t = {"q": _normal(g, (b, sq, h, d), qs, dt), "k": _normal(g, (b, sk, h, d), qs, dt),
             "v": _normal(g, (b, sk, h, d), 1.0, dt)}
    if case["rel"]:
        t["table"] = _normal(g, (32, h), 0.5, dt)
    mask = _padding(g, b, sk).to(dt) if case["mask"] else None
    return t, mask, _normal(g, (b, sq, h, d), 1.0, dt)


def _mlp_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    t, h, f = case["tokens"], case["hidden"], case["inner"]
    return {"x": _normal(g, (t, h), 1.0, dt), "w1": _normal(g, (f, h), h ** -0.5, dt),
            "b1": _normal(g, (f,), 0.1, dt), "w2": _normal(g, (h, f), f ** -0.5, dt),
            "b2": _normal(g, (h,), 0.1, dt), "dy": _normal(g, (t, h), 1.0, dt)}


def _norm_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    t, h = case["tokens"], case["hidden"]
    got = {"x": _normal(g, (t, h), 1.0, dt, 0.1), "w": _normal(g, (h,), 0.1, dt, 1.0),
           "dy": _normal(g, (t, h), 1.0, dt)}
    if case["form"] != "rms":
        got["b"] = _normal(g, (h,), 0.1, dt)
    if case["form"] == "dropout_add":
        got["bias"] = _normal(g, (h,), 0.1, dt)
        got["res"] = _normal(g, (t, h), 1.0, dt)
    return got


def _ce_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    t, v = case["tokens"], case["vocab"]
    logits = torch.empty((t, v), dtype=dt, device=DEV)
    for i in range(0, t, 1024):
        logits[i:i + 1024] = _normal(g, (min(1024, t - i), v), 2.0, dt)
    labels = torch.randint(0, v, (t,), generator=g, device=DEV)
    drop = torch.rand((t,), generator=g, device=DEV) >= case["keep"]
    labels = labels.masked_fill(drop, -100)
    labels[0] = 7
    return logits, labels, torch.rand((t,), generator=g, device=DEV) / t


def _decode_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    b, n, s, h, d = (case[k] for k in ("batch", "new", "past", "heads", "dim"))
    w = h * d
    return {"x": _normal(g, (b, n, w), 1.0, dt), "k": _normal(g, (b, s, h, d), 1.0, dt),
            "v": _normal(g, (b, s, h, d), 1.0, dt),
            "wqkv": _normal(g, (3 * w, w), w ** -0.5, dt), "bqkv": _normal(g, (3 * w,), 0.1, dt),
            "wo": _normal(g, (w, w), w ** -0.5, dt), "bo": _normal(g, (w,), 0.1, dt)}


def _bert_inputs(case, seed):
    """Weights by parameter name, token ids and labels of a masked-LM BERT."""
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    h, f, v = case["hidden"], case["inner"], case["vocab"]
    w = {}

    def linear(name, n, k):
        w[name + ".weight"] = _normal(g, (n, k), k ** -0.5, dt)
        w[name + ".bias"] = _normal(g, (n,), 0.02, dt)

    def norm(name):
        w[name + ".weight"] = _normal(g, (h,), 0.05, dt, 1.0)
        w[name + ".bias"] = _normal(g, (h,), 0.02, dt)

    for name, n in (("word", v), ("position", 512), ("token_type", 2)):
        w["bert.embeddings.%s_embeddings.weight" % name] = _normal(g, (n, h), 0.05, dt)
    norm("bert.embeddings.LayerNorm")
    for i in range(case["layers"]):
        at = "bert.encoder.layer.%d." % i
        linear(at + "attention.self.self_attn.qkv", 3 * h, h)
        linear(at + "attention.output.dense", h, h)
        norm(at + "attention.output.LayerNorm")
        linear(at + "intermediate.dense", f, h)
        linear(at + "output.dense", h, f)
        norm(at + "output.LayerNorm")
    linear("cls.predictions.transform.dense", h, h)
    norm("cls.predictions.transform.LayerNorm")
    w["cls.predictions.bias"] = _normal(g, (v,), 0.02, dt)
    shape = (case["batch"], case["seq"])
    ids = torch.randint(0, v, shape, generator=g, device=DEV)
    labels = ids.masked_fill(torch.rand(shape, generator=g, device=DEV) >= 0.15, -100)
    labels[0, 0] = ids[0, 0]
    return w, ids, labels


def _bert_engine(case, weights):
    p = case.get("p", 0.0)
    cfg = BertConfig(vocab_size=case["vocab"], hidden_size=case["hidden"],
                     num_hidden_layers=case["layers"], num_attention_heads=case["heads"],
                     intermediate_size=case["inner"], hidden_dropout_prob=p,
                     attention_probs_dropout_prob=p)
    with slapo.init_empty_weights():
        model = BertForMaskedLM(cfg)
    sch = slapo.model_schedule.apply_schedule(
        model, "bert", model_config=cfg, bf16=case["dtype"] == "bf16",
        fp16=case["dtype"] == "fp16", ckpt_ratio=0.5 if case["kind"] == "step" else 0.0)
    engine, _ = slapo.build(sch, target="native", init_weights=_no_init,
                            config={"lr": 1e-4, "weight_decay": 0.01, "clip_grad": 1.0})
    left = set(weights)
    with torch.no_grad():
        for name, param in engine.model.named_parameters():
            name = name.replace("predictions.decoder.bias", "predictions.bias")
            name = re.sub(r"(layer\.\d+)\.mod\.", r"\1.", name)      # a checkpointed layer
            param.copy_(weights[name])
            left.discard(name)
    if left:
        raise RuntimeError("parameters without a place: %s" % sorted(left))
    engine.refresh_master_from_params()
    return engine


def _no_init(module, path=None):
    pass


# --------------------------------------------------------------------------- #
def prepare(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    state = {"case": case, "seed": int(seed)}
    if kind == "attn":
        t, mask, dout = _attn_inputs(case, seed)
        op = FlashAttentionOp("auto", case["causal"], 1.0 if case["rel"] else None,
                              rel_bidirectional=not case["causal"])
        state.update(t=t, mask=mask, dout=dout, op=op.train(case["train"]))
        for x in t.values():
            x.requires_grad_(case["train"])
    elif kind == "mlp":
        t = _mlp_inputs(case, seed)
        mod = FusedMLP(case["hidden"], case["inner"], case["act"], case["p"], device=DEV, dtype=dt)
        with torch.no_grad():
            for dst, src in ((mod.fc_in.weight, "w1"), (mod.fc_in.bias, "b1"),
                             (mod.fc_out.weight, "w2"), (mod.fc_out.bias, "b2")):
                dst.copy_(t[src])
        state.update(x=t["x"].requires_grad_(), dy=t["dy"], mod=mod.train())
    elif kind == "norm":
        t, h = _norm_inputs(case, seed), case["hidden"]
        if case["form"] == "dropout_add":
            mod = FusedDropoutAddLayerNorm(h, case["p"], 1e-12, device=DEV, dtype=dt)
            state.update(res=t["res"].requires_grad_(), bias=t["bias"].requires_grad_())
        elif case["form"] == "layer":
            mod = FusedLayerNorm(h, 1e-5, device=DEV, dtype=dt)
        else:
            mod = FusedRMSNorm(h, 1e-6, device=DEV, dtype=dt)
        with torch.no_grad():
            mod.weight.copy_(t["w"])
            if "b" in t:
                mod.bias.copy_(t["b"])
        state.update(x=t["x"].requires_grad_(), dy=t["dy"], mod=mod.train())
    elif kind == "ce":
        logits, labels, coef = _ce_inputs(case, seed)
        state.update(logits=logits.requires_grad_(), labels=labels, coef=coef,
                     mod=ParallelCrossEntropy())
    elif kind == "decode":
        t = _decode_inputs(case, seed)
        mod = FlashAttention(case["heads"] * case["dim"], case["heads"], fused_qkv=True,
                             output_proj=True, causal=True, device=DEV, dtype=dt).eval()
        adopt_native_linears(mod)      # what the native build does to every linear layer
        with torch.no_grad():
            for dst, src in ((mod.qkv.weight, "wqkv"), (mod.qkv.bias, "bqkv"),
                             (mod.out_proj.weight, "wo"), (mod.out_proj.bias, "bo")):
                dst.copy_(t[src])
        state.update(x=t["x"], past=(t["k"], t["v"]), mod=mod)
    else:
        weights, ids, labels = _bert_inputs(case, seed)
        engine = _bert_engine(case, weights)
        engine.model.train(kind == "step")
        state.update(engine=engine, ids=ids, labels=labels)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if case.get("p"):
        # a step that can be replayed: its dropout masks follow from the seed
        torch.cuda.manual_seed(state["seed"])
    if kind == "attn":
        t, op, p = state["t"], state["op"], case["p"]
        with torch.set_grad_enabled(case["train"]):
            if "qkv" in t:
                out = op.forward_packed(t["qkv"], state["mask"], p)
            else:
                out = op(t["q"], t["k"], t["v"], state["mask"], p if case["train"] else 0.0,
                         rel_bias_table=t.get("table"))
        if not case["train"]:
            return {"out": out}
        grads = torch.autograd.grad(out, list(t.values()), state["dout"])
        return {"out": out.detach(), **{"d" + k: x for k, x in zip(t, grads)}}
    if kind == "mlp":
        m = state["mod"]
        wrt = [state["x"], m.fc_in.weight, m.fc_in.bias, m.fc_out.weight, m.fc_out.bias]
        y = m(state["x"])
        return [y.detach(), *torch.autograd.grad(y, wrt, state["dy"])]
    if kind == "norm":
        m = state["mod"]
        wrt = [state["x"], m.weight]
        if case["form"] != "rms":
            wrt.append(m.bias)
        if case["form"] == "dropout_add":
            wrt += [state["res"], state["bias"]]
            y = m(state["x"], state["res"], state["bias"])
        else:
            y = m(state["x"])
        return [y.detach(), *torch.autograd.grad(y, wrt, state["dy"])]
    if kind == "ce":
        loss = state["mod"](state["logits"], state["labels"])
        return [loss.detach(), *torch.autograd.grad(loss, [state["logits"]], state["coef"])]
    if kind == "decode":
        with torch.no_grad():
            out, present = state["mod"](state["x"], layer_past=state["past"], use_cache=True)
        return [out, present[0], present[1]]
    engine = state["engine"]
    if kind == "infer":
        with torch.no_grad():
            return engine(state["ids"])["logits"]
    logits = engine(state["ids"])["logits"]
    loss = mlm_loss(logits, state["labels"])
    engine.backward(loss)
    engine.step()
    return {"loss": loss.detach(), "logits": logits.detach(), "moments": engine.exp_avg,
            "params": engine.flat_param}


# --------------------------------------------------------------------------- #
def _seen(case):
    """Query-key pairs that attention has to look at (per batch and head)."""
    sq, sk = case["sq"], case["sk"]
    return sq * (sq + 1) / 2 if case["causal"] else sq * sk


def _bert_work(case):
    h, f, v, n = case["hidden"], case["inner"], case["vocab"], case["layers"]
    t = case["batch"] * case["seq"]
    params = n * (4 * h * h + 2 * h * f + 9 * h + f) + (v + 514) * h + h * h + v + 4 * h
    layer = 2 * t * (4 * h * h + 2 * h * f) + 4 * t * case["seq"] * h
    return t, params, n * layer + 2 * t * h * (h + v)


def work(case):
    kind = case["kind"]
    e = 4 if case["dtype"] == "fp32" else 2
    if kind == "attn":
        b, h, d = case["batch"], case["heads"], case["dim"]
        one = b * h * d * e
        pairs = b * h * d * _seen(case)
        if not case["train"]:
            return {"bytes": one * (2 * case["sq"] + 2 * case["sk"]), "flops": 4 * pairs}
        # q, dO, out, dQ on one side; k, v, dK, dV on the other; 2 + 5 products
        return {"bytes": one * (4 * case["sq"] + 4 * case["sk"]), "flops": 14 * pairs}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["inner"]
        return {"bytes": e * (4 * t * h + 4 * h * f + 2 * (h + f)), "flops": 12 * t * h * f}
    if kind == "norm":
        t, h = case["tokens"], case["hidden"]
        n = 6 if case["form"] == "dropout_add" else 4
        return {"bytes": e * n * t * h, "flops": 0}
    if kind == "ce":
        kept = case["tokens"] * case["keep"]
        return {"bytes": e * (kept + case["tokens"]) * case["vocab"], "flops": 0}
    if kind == "decode":
        b, n, s, h, d = (case[k] for k in ("batch", "new", "past", "heads", "dim"))
        w = h * d
        cache = 2 * b * w * (2 * s + n)        # read the old one, write the new one
        return {"bytes": e * (4 * w * w + 4 * w + 2 * b * n * w + cache),
                "flops": 8 * b * n * w * w + 4 * b * n * w * (s + n)}
    t, params, flops = _bert_work(case)
    logits = t * case["vocab"] * e
    if kind == "infer":
        return {"bytes": e * params + logits, "flops": flops}
    # weights read and written, fp32 master and moments read and written, logits returned
    return {"bytes": params * (2 * e + 24) + logits, "flops": 3 * flops}


def tolerance(case):
    """About four times the error against ``exact`` that the 16-bit roundings of inputs,
    intermediates and results leave; 32-bit sums in another order for fp32."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    if case["kind"] == "step":
        return {"rel": 0.03}
    bf16 = 0.03 if case["kind"] == "infer" else 0.014     # measured: 0.0076 and up to 0.0034
    return {"rel": bf16 if case["dtype"] == "bf16" else bf16 / 7}


# --------------------------------------------------------------------------- #
def _keep(rows, cols, seed, p, span=None):
    """Keep mask [rows, cols] of one dropout call with a fresh generator.  A group of 16
    elements is one Philox call; a row takes ``span`` groups, or the elements run on from row
    to row (None).  Returns the mask and the kept values' factor."""
    thr = min(max(int(p * 128.0 + 0.5), 0), 127)
    total = rows * span if span else -(-rows * cols // 16)
    parts = []
    low32 = 0xFFFFFFFF

    def mul(const, x):
        low, high = const * (x & 0xFFFF), const * (x >> 16)
        low = low + ((high & 0xFFFF) << 16)
        return low & low32, (high >> 16) + (low >> 32)

    for at in range(0, total, 1 << 22):
        i = torch.arange(at, min(total, at + (1 << 22)), device=DEV)
        c = [torch.zeros_like(i), torch.zeros_like(i), i & low32, i >> 32]
        k0, k1 = seed & low32, (seed >> 32) & low32
        for _ in range(7):
            l0, h0 = mul(0xD2511F53, c[0])
            l1, h1 = mul(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & low32, (k1 + 0xBB67AE85) & low32
        words = torch.stack(c, dim=1)
        byte = torch.stack([(words >> (8 * j)) & 0x7F for j in range(4)], dim=2)
        parts.append((byte >= thr).reshape(-1))
    keep = torch.cat(parts)
    keep = keep.view(rows, span * 16)[:, :cols] if span else keep[:rows * cols].view(rows, cols)
    return keep, 128.0 / (128.0 - thr)


def _buckets(sq, sk, bidirectional):
    """T5's bucket of key - query (32 buckets, distances up to 128)."""
    rel = torch.arange(sk, device=DEV)[None, :] - (torch.arange(sq, device=DEV)[:, None] + sk - sq)
    n, at = 32, torch.zeros_like(rel)
    if bidirectional:
        n = 16
        at = (rel > 0).long() * n
        rel = rel.abs()
    else:
        rel = (-rel).clamp(min=0)
    near = n // 2
    far = near + (torch.log(rel.float().clamp(min=1) / near) / math.log(128 / near)
                  * (n - near)).long()
    return at + torch.where(rel < near, rel, far.clamp(max=n - 1))


def _attention(q, k, v, causal, scale, mask=None, bias=None, keep=None, factor=1.0):
    """[B, S, H, D] attention; ``keep`` [B, H, Sq, Sk]."""
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    if bias is not None:
        s = s + bias
    if mask is not None:
        s = s + mask
    if causal:
        sq, sk = s.shape[-2:]
        ahead = torch.ones(sq, sk, dtype=torch.bool, device=DEV).triu(sk - sq + 1)
        s = s.masked_fill(ahead, float("-inf"))
    p = torch.softmax(s, dim=-1)
    if keep is not None:
        p = p * keep * factor
    return torch.einsum("bhqk,bkhd->bqhd", p, v)


def _exact_attn(case, seed):
    t, mask, dout = _attn_inputs(case, seed)
    b, sq, sk, h, d = (case[k] for k in ("batch", "sq", "sk", "heads", "dim"))
    scale = 1.0 if case["rel"] else d ** -0.5
    p = case["p"] if case["train"] else 0.0
    outs, grads, dtable = [], {k: [] for k in t}, None
    table = t["table"].double().requires_grad_(case["train"]) if case["rel"] else None
    keep, factor = None, 1.0
    if p:
        keep, factor = _keep(b * h * sq, sk, seed, p, span=-(-sk // 16))
        keep = keep.reshape(b, h, sq, sk)
    for i in range(b):
        own = {k: x[i:i + 1].double().requires_grad_(case["train"]) for k, x in t.items()
               if k != "table"}
        q, k, v = own["qkv"].unbind(3) if "qkv" in own else (own["q"], own["k"], own["v"])
        bias = None
        if table is not None:
            bias = table[_buckets(sq, sk, not case["causal"])].permute(2, 0, 1)[None]
        o = _attention(q, k, v, case["causal"], scale,
                       None if mask is None else mask[i:i + 1].double(), bias,
                       None if keep is None else keep[i:i + 1], factor)
        outs.append(o.detach())
        if case["train"]:
            wrt = list(own.values()) + ([table] if table is not None else [])
            got = torch.autograd.grad(o, wrt, dout[i:i + 1].double())
            for key, x in zip(own, got):
                grads[key].append(x)
            if table is not None:
                dtable = got[-1] if dtable is None else dtable + got[-1]
    if not case["train"]:
        return {"out": torch.cat(outs)}
    out = {"out": torch.cat(outs)}
    for key in t:
        out["d" + key] = dtable if key == "table" else torch.cat(grads[key])
    return out


def _act(x, name):
    if name == "relu":
        return F.relu(x)
    return F.gelu(x, approximate="none" if name == "gelu" else "tanh")


def _exact_mlp(case, seed):
    t = {k: x.double() for k, x in _mlp_inputs(case, seed).items()}
    wrt = [t[k].requires_grad_() for k in ("x", "w1", "b1", "w2", "b2")]
    y = _act(F.linear(t["x"], t["w1"], t["b1"]), case["act"])
    y = F.linear(y, t["w2"], t["b2"])
    if case["p"]:
        keep, factor = _keep(*y.shape, seed, case["p"])
        y = y * keep * factor
    return [y.detach(), *torch.autograd.grad(y, wrt, t["dy"])]


def _exact_norm(case, seed):
    t = {k: x.double() for k, x in _norm_inputs(case, seed).items()}
    wrt = [t[k].requires_grad_() for k in ("x", "w", "b", "res", "bias") if k in t]
    z, h = t["x"], case["hidden"]
    if case["form"] == "rms":
        y = z * torch.rsqrt(z.square().mean(-1, keepdim=True) + 1e-6) * t["w"]
    elif case["form"] == "layer":
        y = F.layer_norm(z, (h,), t["w"], t["b"], 1e-5)
    else:
        z = z + t["bias"]
        if case["p"]:
            keep, factor = _keep(*z.shape, seed, case["p"])
            z = z * keep * factor
        y = F.layer_norm(z + t["res"], (h,), t["w"], t["b"], 1e-12)
    return [y.detach(), *torch.autograd.grad(y, wrt, t["dy"])]


def _exact_ce(case, seed):
    logits, labels, coef = _ce_inputs(case, seed)
    loss, grad = [], []
    for i in range(0, case["tokens"], 1024):
        x = logits[i:i + 1024].double()
        lab = labels[i:i + 1024]
        real = lab != -100
        logp = torch.log_softmax(x, dim=-1)
        at = lab.clamp(min=0)[:, None]
        loss.append(-logp.gather(1, at)[:, 0] * real)
        g = logp.exp().scatter_add_(1, at, -torch.ones_like(at, dtype=torch.float64))
        grad.append(g * (coef[i:i + 1024].double() * real)[:, None])
    return [torch.cat(loss), torch.cat(grad)]


def _exact_decode(case, seed):
    t = {k: x.double() for k, x in _decode_inputs(case, seed).items()}
    b, n, h, d = (case[k] for k in ("batch", "new", "heads", "dim"))
    qkv = F.linear(t["x"], t["wqkv"], t["bqkv"]).view(b, n, h, 3, d)
    k = torch.cat([t["k"], qkv[..., 1, :]], dim=1)
    v = torch.cat([t["v"], qkv[..., 2, :]], dim=1)
    o = _attention(qkv[..., 0, :], k, v, True, d ** -0.5).reshape(b, n, h * d)
    return [F.linear(o, t["wo"], t["bo"]), k, v]


def _exact_infer(case, seed):
    weights, ids, _ = _bert_inputs(case, seed)
    w = {k: x.double() for k, x in weights.items()}
    h, n = case["hidden"], case["heads"]

    def linear(name, x):
        return F.linear(x, w[name + ".weight"], w[name + ".bias"])

    def norm(name, x):
        return F.layer_norm(x, (h,), w[name + ".weight"], w[name + ".bias"], 1e-12)

    emb = "bert.embeddings.%s_embeddings.weight"
    x = w[emb % "word"][ids] + w[emb % "position"][:case["seq"]] + w[emb % "token_type"][0]
    x = norm("bert.embeddings.LayerNorm", x)
    for i in range(case["layers"]):
        at = "bert.encoder.layer.%d." % i
        qkv = linear(at + "attention.self.self_attn.qkv", x).view(*ids.shape, n, 3, h // n)
        a = _attention(*qkv.unbind(3), False, (h // n) ** -0.5).reshape(x.shape)
        x = norm(at + "attention.output.LayerNorm", x + linear(at + "attention.output.dense", a))
        f = F.gelu(linear(at + "intermediate.dense", x))
        x = norm(at + "output.LayerNorm", x + linear(at + "output.dense", f))
    x = norm("cls.predictions.transform.LayerNorm",
             F.gelu(linear("cls.predictions.transform.dense", x)))
    return F.linear(x, w[emb % "word"], w["cls.predictions.bias"])


def exact(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind == "step":
        return None     # its embedding dropout is PyTorch's own, drawn from the same generator
    return {"attn": _exact_attn, "mlp": _exact_mlp, "norm": _exact_norm, "ce": _exact_ce,
            "decode": _exact_decode, "infer": _exact_infer}[kind](case, seed)
