"""The work this framework is timed on: calls through its public entry points, at the sizes users bring.

A case is a dict of plain values with a `kind`:

* `decode`     one cached-attention step, `flash_decoding_with_fusing_bias`
* `layer`      one encoder self-attention module in float32, `T5FlashAttention`
* `attention`  the dense operator, `flash_attention_with_fusing_bias`, forward
* `varlen`     the packed-sequence operator, `flash_attention_with_fusing_bias_varlen`, forward
* `local`      block-local attention (`local_block=`), forward
* `gradient`   the dense operator, forward and backward (q, k, v and the bias table)
* `seq2seq`    `T5ForConditionalGeneration` forward for inference, with or without a padding mask
* `generate`   `T5ForConditionalGeneration.greedy_decode`: cached keys, one captured step per token
* `train`      forward, loss and backward of a small encoder-decoder on a padded batch

Weights are random with the variances of a T5 initialisation, the projections into the residual stream
scaled down by depth; activations are N(0, 1) and bias tables N(0, 0.1).
"""
import math
import random

import torch

import turbot5_b200 as t5b
from turbot5_b200.modules import T5FlashAttention
from turbot5_b200.t5 import T5ForConditionalGeneration, T5StackConfig

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BUCKETS, _MAX_DISTANCE = 32, 128
_VOCAB = 32128

_MODELS = {
    # d_model, heads, d_kv, d_ff, encoder layers, decoder layers, feed-forward
    "small": (512, 8, 64, 1024, 6, 6, "gated-gelu"),
    "base": (768, 12, 64, 2048, 12, 12, "gated-gelu"),
    "large": (1024, 16, 64, 4096, 24, 24, "relu"),
}


def listed():
    return [
        # One sequence, one new token early in a generation: a few hundred cached keys, all latency.
        dict(name="decode_one_sequence", kind="decode", B=1, H=12, N=512, used=200, self_attention=True, dtype="bf16"),
        # Cross attention of one large-shaped decoder layer for a full serving batch: the K/V stream.
        dict(name="decode_serving_batch", kind="decode", B=64, H=16, N=8192, used=8192, self_attention=False,
             dtype="bf16"),
        # The float32 layer that the module is checked on: short inputs, full precision.
        dict(name="layer_float32", kind="layer", B=2, L=512),
        # Encoder self-attention of an ordinary batch of documents.
        dict(name="attention_1k", kind="attention", B=16, H=12, M=1024, N=1024, D=64, causal=False, bias=True,
             dtype="bf16"),
        # Encoder self-attention of long documents: the headline size.
        dict(name="attention_8k", kind="attention", B=2, H=12, M=8192, N=8192, D=64, causal=False, bias=True,
             dtype="bf16"),
        # Decoder prefill with the wide heads of the largest T5 sizes, at a length that is no multiple of a tile.
        dict(name="attention_causal_d128", kind="attention", B=2, H=16, M=3000, N=3000, D=128, causal=True, bias=True,
             dtype="fp16"),
        # A batch of documents of every length, packed.
        dict(name="varlen_mixed", kind="varlen", count=32, shortest=128, longest=4096, lengths=1, H=12, D=64,
             dtype="bf16"),
        # One very long document with LongT5-style block-local attention.
        dict(name="local_64k", kind="local", B=1, H=12, L=65536, block=512, dtype="bf16"),
        # Attention core of a training step on long documents.
        dict(name="gradient_8k", kind="gradient", B=2, H=12, L=8192, D=64, causal=False, dtype="bf16"),
        # Inference on a padded batch: prompts of uneven length, teacher-forced targets.
        dict(name="seq2seq_padded", kind="seq2seq", model="base", B=16, L=1024, targets=128, padded=True, lengths=2),
        # Greedy generation against encoder states that are already there.
        dict(name="generate_large", kind="generate", model="large", B=16, L=1024, steps=32),
        # A fine-tuning step of a small model on a padded batch.
        dict(name="train_small", kind="train", model="small", B=8, L=512, targets=128, lengths=3),
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    kind = rng.choice(("decode", "decode", "layer", "attention", "attention", "varlen", "local", "gradient",
                       "gradient", "seq2seq", "generate", "train"))
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
    H = rng.choice((8, 12, 16))
    if kind == "decode":
        N = _between(rng, 64, 8192)
        return dict(kind=kind, B=_between(rng, 1, 64), H=H, N=N, used=rng.randint(max(1, N // 3), N),
                    self_attention=rng.random() < 0.5, dtype=dtype)
    if kind == "layer":
        return dict(kind=kind, B=_between(rng, 1, 4), L=_between(rng, 64, 1024))
    if kind == "attention":
        D = rng.choice((64, 64, 64, 128, 32))
        M = _between(rng, 128, 8192)
        cross = rng.random() < 0.25
        N = _between(rng, 128, 8192) if cross else M
        B = max(1, min(_between(rng, 1, 32), int(2 * 12 * 8192 * 8192 * 64 / (H * M * N * D))))
        return dict(kind=kind, B=B, H=H, M=M, N=N, D=D, causal=not cross and rng.random() < 0.4, bias=not cross,
                    dtype=dtype)
    if kind == "varlen":
        return dict(kind=kind, count=_between(rng, 2, 32), shortest=rng.choice((16, 64, 128)),
                    longest=_between(rng, 256, 4096), lengths=rng.randrange(1 << 20), H=min(H, 12), D=64, dtype=dtype)
    if kind == "local":
        return dict(kind=kind, B=1, H=min(H, 12), L=_between(rng, 2048, 65536), block=rng.choice((128, 256, 512)),
                    dtype=dtype)
    if kind == "gradient":
        D = rng.choice((64, 64, 128))
        L = _between(rng, 128, 8192)
        B = max(1, min(_between(rng, 1, 16), int(2 * 12 * 8192 * 8192 * 64 / (H * L * L * D))))
        return dict(kind=kind, B=B, H=H, L=L, D=D, causal=rng.random() < 0.4, dtype=dtype)
    if kind == "seq2seq":
        return dict(kind=kind, model="base", B=_between(rng, 1, 16), L=_between(rng, 64, 1024),
                    targets=_between(rng, 8, 128), padded=rng.random() < 0.6, lengths=rng.randrange(1 << 20))
    if kind == "generate":
        return dict(kind=kind, model=rng.choice(("small", "base", "large")), B=_between(rng, 1, 16),
                    L=_between(rng, 64, 1024), steps=_between(rng, 8, 32))
    return dict(kind=kind, model="small", B=_between(rng, 1, 8), L=_between(rng, 64, 512),
                targets=_between(rng, 16, 128), lengths=rng.randrange(1 << 20))


# ---- sizes that follow from a case

def _varlen_lengths(case):
    r = random.Random(case["lengths"])
    return [r.randint(case["shortest"], case["longest"]) for _ in range(case["count"])]


def _prompt_lengths(case):
    """Valid tokens of each prompt of a padded batch: between an eighth of the width and all of it."""
    if not case.get("padded", True):
        return [case["L"]] * case["B"]
    r = random.Random(case["lengths"])
    return [r.randint(max(1, case["L"] // 8), case["L"]) for _ in range(case["B"])]


# ---- inputs, weights and handles

def _normal(g, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _heads(g, B, H, L, D, dtype, std=1.0):
    """(B, H, L, D) view of token-major rows, as a projection gives it."""
    return _normal(g, (B, L, H, D), dtype, std).transpose(1, 2)


def _table(g, H, dtype):
    return _normal(g, (_BUCKETS, H), dtype, 0.1)


def _config(name, dropout=0.0):
    d_model, heads, d_kv, d_ff, enc, dec, ff = _MODELS[name]
    return T5StackConfig(vocab_size=_VOCAB, d_model=d_model, d_kv=d_kv, d_ff=d_ff, num_layers=enc,
                         num_decoder_layers=dec, num_heads=heads, relative_attention_num_buckets=_BUCKETS,
                         relative_attention_max_distance=_MAX_DISTANCE, dropout_rate=dropout, feed_forward_proj=ff)


def _init_std(name, p, cfg):
    if p.dim() == 1:
        return 0.0
    leaf = name.split(".")[-2]
    into_residual = (2 * cfg.num_decoder_layers) ** -0.5
    if leaf == "q":
        return (cfg.d_model * cfg.d_kv) ** -0.5
    if leaf == "o":
        return (cfg.num_heads * cfg.d_kv) ** -0.5 * into_residual
    if leaf == "wo":
        return cfg.d_ff ** -0.5 * into_residual
    if leaf == "shared":
        return 1.0
    return cfg.d_model ** -0.5


def _model(name, g, encoder=True):
    cfg = _config(name)
    if not encoder:
        cfg.num_layers = 1          # generation from given encoder states: the encoder is not called
    with torch.device("meta"):
        model = T5ForConditionalGeneration(cfg)
    model = model.to(torch.bfloat16).to_empty(device="cuda")
    with torch.no_grad():
        for pname, p in model.named_parameters():
            std = _init_std(pname, p, cfg)
            p.fill_(1.0) if p.dim() == 1 else p.normal_(0.0, std, generator=g)
    return model


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    dtype = _DTYPES[case.get("dtype", "bf16")]
    s = dict(case=case)
    if kind == "decode":
        B, H, N = case["B"], case["H"], case["N"]
        s["q"] = _normal(g, (B, H, 1, 64), dtype)
        s["k"], s["v"] = _normal(g, (B, H, N, 64), dtype), _normal(g, (B, H, N, 64), dtype)
        s["table"] = _table(g, H, dtype) if case["self_attention"] else None
    elif kind == "layer":
        cfg = _config("small")
        layer = T5FlashAttention(cfg, has_relative_attention_bias=True).cuda()
        with torch.no_grad():
            for p in layer.parameters():
                p.normal_(0.0, 0.05, generator=g)
            layer.relative_attention_bias.weight.normal_(0.0, 0.1, generator=g)
        s["layer"] = layer
        s["hidden"] = _normal(g, (case["B"], case["L"], cfg.d_model), torch.float32)
    elif kind == "attention":
        B, H, M, N, D = (case[n] for n in ("B", "H", "M", "N", "D"))
        std = (64 / max(D, 64)) ** 0.5
        s["q"], s["k"] = _heads(g, B, H, M, D, dtype, std), _heads(g, B, H, N, D, dtype, std)
        s["v"] = _heads(g, B, H, N, D, dtype)
        s["table"] = _table(g, H, dtype) if case["bias"] else None
    elif kind == "varlen":
        lens, H, D = _varlen_lengths(case), case["H"], case["D"]
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        s["q"], s["k"], s["v"] = (_normal(g, (cu[-1], H, D), dtype) for _ in range(3))
        s["table"] = _table(g, H, dtype)
        s["cu"], s["max"] = torch.tensor(cu, dtype=torch.int32, device="cuda"), max(lens)
    elif kind == "local":
        s["q"], s["k"], s["v"] = (_heads(g, case["B"], case["H"], case["L"], 64, dtype) for _ in range(3))
        s["table"] = _table(g, case["H"], dtype)
    elif kind == "gradient":
        B, H, L, D = (case[n] for n in ("B", "H", "L", "D"))
        std = 0.5 * (64 / D) ** 0.5
        q, k, v = _heads(g, B, H, L, D, dtype, std), _heads(g, B, H, L, D, dtype, std), _heads(g, B, H, L, D, dtype)
        s["inputs"] = [t.requires_grad_() for t in (q, k, v, _table(g, H, dtype))]
        s["dout"] = _heads(g, B, H, L, D, dtype)
    elif kind == "seq2seq":
        s["model"] = _model(case["model"], g)
        s["ids"] = torch.randint(0, _VOCAB, (case["B"], case["L"]), generator=g, device="cuda")
        s["targets"] = torch.randint(0, _VOCAB, (case["B"], case["targets"]), generator=g, device="cuda")
        s["mask"] = _mask(case) if case["padded"] else None
    elif kind == "generate":
        model = _model(case["model"], g, encoder=False)
        # A trained model is sure of most of its next tokens; random heads would make every step a near tie.
        # Each token's embedding is the head's row of another token, which then leads the logits by a margin.
        with torch.no_grad():
            order = torch.randperm(_VOCAB, generator=g, device="cuda")
            model.lm_head.weight.copy_(model.shared.weight[order])
        s["model"] = model
        s["memory"] = _normal(g, (case["B"], case["L"], model.cfg.d_model), torch.bfloat16)
    else:
        model = _model(case["model"], g)
        # gradients in one buffer, as data-parallel training keeps them
        params = list(model.parameters())
        flat = torch.zeros(sum(p.numel() for p in params), dtype=torch.bfloat16, device="cuda")
        at = 0
        for p in params:
            p.grad = flat[at:at + p.numel()].view_as(p)
            at += p.numel()
        s["model"], s["grads"] = model, flat
        s["ids"] = torch.randint(0, _VOCAB, (case["B"], case["L"]), generator=g, device="cuda")
        s["targets"] = torch.randint(0, _VOCAB, (case["B"], case["targets"]), generator=g, device="cuda")
        s["labels"] = torch.randint(0, _VOCAB, (case["B"] * case["targets"],), generator=g, device="cuda")
        s["mask"] = _mask(case)
    return s


def _mask(case):
    lens = torch.tensor(_prompt_lengths(case), device="cuda")
    return (torch.arange(case["L"], device="cuda")[None, :] < lens[:, None]).to(torch.int64)


# ---- one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gradient":
        out = t5b.flash_attention_with_fusing_bias(*s["inputs"], causal=case["causal"], sm_scale=1.0,
                                                   NUM_BUCKETS=_BUCKETS, MAX_DISTANCE=_MAX_DISTANCE)
        return (out,) + torch.autograd.grad(out, s["inputs"], s["dout"])
    if kind == "train":
        s["grads"].zero_()
        logits = s["model"](s["ids"], s["targets"], attention_mask=s["mask"])
        loss = torch.nn.functional.cross_entropy(logits.flatten(0, 1).float(), s["labels"])
        loss.backward()
        return loss.detach(), s["grads"]
    with torch.no_grad():
        if kind == "decode":
            own = case["self_attention"]
            return t5b.flash_decoding_with_fusing_bias(s["q"], s["k"], s["v"], s["table"], causal=own, sm_scale=1.0,
                                                       NUM_BUCKETS=_BUCKETS, MAX_DISTANCE=_MAX_DISTANCE,
                                                       kv_len=case["used"], q_pos_offset=None if own else 0)
        if kind == "layer":
            return s["layer"](s["hidden"])[0]
        if kind == "attention":
            return t5b.flash_attention_with_fusing_bias(s["q"], s["k"], s["v"], s["table"], causal=case["causal"],
                                                        sm_scale=1.0, NUM_BUCKETS=_BUCKETS,
                                                        MAX_DISTANCE=_MAX_DISTANCE,
                                                        q_pos_offset=None if case["bias"] else 0)
        if kind == "varlen":
            return t5b.flash_attention_with_fusing_bias_varlen(s["q"], s["k"], s["v"], s["table"], s["cu"], s["cu"],
                                                               s["max"], s["max"], causal=False, sm_scale=1.0,
                                                               NUM_BUCKETS=_BUCKETS, MAX_DISTANCE=_MAX_DISTANCE)
        if kind == "local":
            return t5b.flash_attention_with_fusing_bias(s["q"], s["k"], s["v"], s["table"], sm_scale=1.0,
                                                        NUM_BUCKETS=_BUCKETS, MAX_DISTANCE=_MAX_DISTANCE,
                                                        local_block=case["block"])
        if kind == "seq2seq":
            return s["model"](s["ids"], s["targets"], attention_mask=s["mask"])
        return s["model"].greedy_decode(s["memory"], case["steps"], use_cuda_graph=True)


# ---- what a pass cannot do without

def _visible(M, N, causal):
    """Query-key pairs of one head (queries at the end of the keys)."""
    return sum(max(0, min(N, N - M + m + 1)) for m in range(M)) if causal else M * N


def _attention_cost(B, H, M, N, D, causal, item):
    return 4.0 * B * H * _visible(M, N, causal) * D, B * H * D * item * (2.0 * M + 2.0 * N)


def _block_params(cfg, decoder):
    inner = cfg.num_heads * cfg.d_kv
    ff = (3 if cfg.feed_forward_proj.startswith("gated") else 2) * cfg.d_model * cfg.d_ff
    return 4 * cfg.d_model * inner + ff, (4 * cfg.d_model * inner if decoder else 0)


def _seq2seq_flops(case):
    """(flops of one forward pass over the valid tokens, parameters without the embedding)."""
    cfg = _config(case["model"])
    inner, B, T = cfg.num_heads * cfg.d_kv, case["B"], case["targets"]
    lens = _prompt_lengths(case)
    tokens = sum(lens)
    enc, _ = _block_params(cfg, False)
    dec, cross = _block_params(cfg, True)
    head = cfg.d_model * cfg.vocab_size
    flops = cfg.num_layers * (2.0 * tokens * enc + 4.0 * inner * sum(n * n for n in lens))
    flops += cfg.num_decoder_layers * (2.0 * B * T * (dec + cross / 2) + 2.0 * tokens * cross / 2
                                       + 4.0 * inner * (B * _visible(T, T, True) + T * tokens))
    flops += 2.0 * B * T * head
    return flops, cfg.num_layers * enc + cfg.num_decoder_layers * (dec + cross) + head


def work(case):
    kind = case["kind"]
    item = 4 if kind == "layer" else 2
    if kind == "decode":
        flops, _ = _attention_cost(case["B"], case["H"], 1, case["used"], 64, False, item)
        return {"bytes": case["B"] * case["H"] * 64.0 * item * (2 * case["used"] + 2), "flops": flops}
    if kind == "layer":
        cfg = _config("small")
        inner, rows = cfg.num_heads * cfg.d_kv, case["B"] * case["L"]
        flops, _ = _attention_cost(case["B"], cfg.num_heads, case["L"], case["L"], cfg.d_kv, False, item)
        return {"bytes": item * (2.0 * rows * cfg.d_model + 4.0 * cfg.d_model * inner),
                "flops": flops + 2.0 * rows * 4 * cfg.d_model * inner}
    if kind == "attention":
        flops, moved = _attention_cost(case["B"], case["H"], case["M"], case["N"], case["D"], case["causal"], item)
        return {"bytes": moved, "flops": flops}
    if kind == "varlen":
        lens = _varlen_lengths(case)
        return {"bytes": 4.0 * sum(lens) * case["H"] * case["D"] * item,
                "flops": 4.0 * case["H"] * case["D"] * sum(n * n for n in lens)}
    if kind == "local":
        rows, block = case["B"] * case["L"], case["block"]
        return {"bytes": 4.0 * rows * case["H"] * 64 * item,
                "flops": 4.0 * rows * case["H"] * min(3 * block, case["L"]) * 64}
    if kind == "gradient":
        flops, moved = _attention_cost(case["B"], case["H"], case["L"], case["L"], case["D"], case["causal"], item)
        return {"bytes": 2.0 * moved, "flops": 3.5 * flops}      # q, k, v, dout in; out, dq, dk, dv out
    if kind == "seq2seq":
        flops, params = _seq2seq_flops(case)
        return {"bytes": item * (params + 1.0 * case["B"] * case["targets"] * _VOCAB), "flops": flops}
    if kind == "generate":
        cfg = _config(case["model"])
        inner, B, L, T = cfg.num_heads * cfg.d_kv, case["B"], case["L"], case["steps"]
        dec, cross = _block_params(cfg, True)
        per_step = cfg.num_decoder_layers * (dec + cross / 2) + cfg.d_model * cfg.vocab_size
        keys = cfg.num_decoder_layers * 2.0 * B * inner
        return {"bytes": item * (T * (per_step + keys * L) + keys * T * (T + 1) / 2 + B * L * cfg.d_model
                                 + cfg.num_decoder_layers * cross / 2),
                "flops": 2.0 * B * T * per_step + 2.0 * B * L * cfg.num_decoder_layers * cross / 2
                + 4.0 * cfg.num_decoder_layers * inner * B * (T * L + T * (T + 1) / 2)}
    flops, params = _seq2seq_flops(case)
    cfg = _config(case["model"])
    return {"bytes": item * (2.0 * params + cfg.d_model * _VOCAB), "flops": 3.0 * flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "layer":
        return {"rel": 3e-5}         # float32 sums, and their differences through one exponential
    if kind in ("seq2seq", "generate"):
        return {"rel": 2e-2}         # bf16 activations through up to 24 blocks; tokens are the same
    if kind in ("gradient", "train"):
        return {"rel": 2e-2}         # bf16 operands in every product of the backward pass
    return {"rel": 1e-2}             # bf16 / fp16 operands, one rounding of the result
