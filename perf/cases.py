"""The work a trainer has this package do, as cases that can be timed and compared.

Four kinds, each through the public operators:

  loss     the fused linear cross-entropy over a vocabulary of 32 k to 152 k: a training step's forward and
           backward (`reduced_linear_cross_entropy`, then the gradient of the hidden states), or the per-token
           losses of a validation batch (`fused_linear_ce` without gradients).  Heads: a frozen dense one
           (LoRA), a frozen 4-bit one (QLoRA), a dense one that is trained too.
  attn     causal flash attention with grouped kv heads: forward and backward, or the forward alone.
  packed   the same over rows that hold several documents (`PackedMask`).
  layer    what the attention wrapper runs between the projections and `o_proj`: q / k norm and rotary
           embedding on the projections' own (B, L, H, d) layout, then attention on the strided views.

Sizes: rows of hidden states from a few dozen (a short prompt, the tail of an epoch) to 8192, hidden sizes
1024 to 4096, sequences of 128 to 16384 tokens, head_dim 64 / 96 / 128; lengths are odd as often as round.
bf16 is what training uses; fp32 losses (never larger than 2048 x 1024 x 32768) are the full-precision option
of small models.
"""
import math

import torch

from mlx_train_perf_b200.attention.api import flash_attention
from mlx_train_perf_b200.attention.prestep import qk_norm_rope
from mlx_train_perf_b200.attention.segments import PackedMask
from mlx_train_perf_b200.core.loss import (IGNORE_INDEX, DenseHead, QuantizedHead, fused_linear_ce,
                                           reduced_linear_cross_entropy)

FLAGSHIP = 8192 * 4096 * 151936            # rows x hidden size x vocabulary of the largest loss
FP32_MOST = 2048 * 1024 * 32768            # and of the largest fp32 one


def _loss(name, n, d, v, head="dense", dtype="bf16", step="train"):
    return {"name": name, "kind": "loss", "n": n, "d": d, "v": v, "head": head, "dtype": dtype, "step": step}


def _attn(name, b, s, hq, hkv, d, step="train", kind="attn", seg_lo=0, seg_hi=0):
    c = {"name": name, "kind": kind, "b": b, "s": s, "hq": hq, "hkv": hkv, "d": d, "step": step}
    if kind == "packed":
        c.update(seg_lo=seg_lo, seg_hi=seg_hi)
    return c


def listed():
    return [
        # one short example on a small model: launches and host work
        _loss("loss_small", 60, 1024, 32768),
        # LoRA micro-batch of about a thousand tokens against a large vocabulary
        _loss("loss_micro", 1000, 4096, 151936),
        # LoRA step on a full batch: the headline workload
        _loss("loss_full", 8192, 4096, 151936),
        # QLoRA step: 4-bit head
        _loss("loss_int4", 2048, 4096, 151936, head="int4"),
        # validation loss of one short batch under a 4-bit head: forward only, per-token results
        _loss("loss_int4_eval", 257, 4096, 151936, head="int4", step="eval"),
        # full fine-tuning of a small model with tied embeddings: the head's gradient too
        _loss("loss_trained_head", 4096, 1024, 151936, head="trained"),
        # full-precision option
        _loss("loss_fp32", 2048, 1024, 32768, dtype="fp32"),
        # short sequences, one micro-batch
        _attn("attn_short", 2, 333, 32, 8, 128),
        # the long-context training shape
        _attn("attn_long", 1, 8192, 32, 8, 128),
        # forward of a validation batch, head_dim 64
        _attn("attn_eval_d64", 2, 2500, 32, 8, 64, step="eval"),
        # packed documents of 128 to 4096 tokens
        _attn("attn_packed", 1, 16384, 32, 8, 128, kind="packed", seg_lo=128, seg_hi=4096),
        # one attention layer of a small model as the wrapper runs it
        _attn("layer", 4, 2048, 16, 8, 128, kind="layer"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loss", "loss", "loss", "attn", "attn", "packed", "layer"])
    if kind == "loss":
        head = rng.choice(["dense", "dense", "int4", "trained"])
        dtype = "fp32" if head == "dense" and rng.random() < 0.2 else "bf16"
        step = "train" if head == "trained" or rng.random() < 0.7 else "eval"
        d = rng.choice([1024, 1536, 2048, 2560, 3072, 4096])
        v = _log_int(rng, 32000, 151936)
        n = _log_int(rng, 32, 8192)
        most = FP32_MOST if dtype == "fp32" else FLAGSHIP * (0.6 if head == "trained" else 1.0)
        n = max(1, min(n, int(most // (d * v))))
        c = _loss("", n, d, v, head, dtype, step)
    else:
        hq, hkv = rng.choice([(32, 8), (16, 8), (16, 16), (12, 4), (14, 2)])
        d = rng.choice([64, 96, 128, 128])
        s = _log_int(rng, 1024 if kind == "packed" else 128, 16384)
        b = rng.randint(1, max(1, min(8, 16384 // s)))
        step = "train" if rng.random() < 0.75 else "eval"
        lo = rng.choice([16, 128, 512])
        c = _attn("", b, s, hq, hkv, d, step, kind, lo, lo + _log_int(rng, 64, 4096))
    del c["name"]
    return c


def _segments(b, s, lo, hi, rng):
    """Segment lengths uniform in [lo, hi] until each row is full, the last one cut; and the two index rows."""
    ids, starts, lengths = torch.empty(b, s, dtype=torch.int32), torch.empty(b, s, dtype=torch.int32), []
    for row in range(b):
        at = k = 0
        while at < s:
            n = min(int(torch.randint(lo, hi + 1, (1,), generator=rng)), s - at)
            ids[row, at:at + n] = k
            starts[row, at:at + n] = at
            lengths.append(n)
            at, k = at + n, k + 1
    return ids, starts, lengths


def _case_segments(case, seed):
    return _segments(case["b"], case["s"], case["seg_lo"], case["seg_hi"], torch.Generator().manual_seed(seed))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = torch.device("cuda")
    train = case["step"] == "train"

    if case["kind"] == "loss":
        n, d, v = case["n"], case["d"], case["v"]
        dtype = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
        hidden = torch.randn(n, d, generator=g, device=dev)
        targets = torch.randint(0, v, (n,), generator=g, device=dev)
        if case["head"] == "int4":
            # codes uniform in [0, 15], scales |N(0, 0.01)|, biases -8 scale
            w_q = torch.randint(-2**31, 2**31, (v, d // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
            scales = (torch.randn(v, d // 64, generator=g, device=dev) * 0.01).abs().to(dtype)
            head = QuantizedHead(w_q, scales, (-8.0 * scales.float()).to(dtype))
        else:
            w = (torch.randn(v, d, generator=g, device=dev, dtype=dtype) * d ** -0.5)
            # a model in training knows some targets well and others not at all: push each row towards its
            # target's weight row, so that the losses run from about ln(v) down to about zero
            hidden += torch.rand(n, 1, generator=g, device=dev) * 20.0 * w[targets].float()
            head = DenseHead(w.requires_grad_(case["head"] == "trained"), trainable=case["head"] == "trained")
        # prompt and padding positions carry no loss
        targets[torch.rand(n, generator=g, device=dev) < 0.03] = IGNORE_INDEX
        hidden = hidden.to(dtype).requires_grad_(train)
        return {"case": case, "hidden": hidden, "head": head, "targets": targets}

    b, s, hq, hkv, d = (case[k] for k in ("b", "s", "hq", "hkv", "d"))

    def rand(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.bfloat16)

    state = {"case": case, "scale": d ** -0.5}
    if case["kind"] == "layer":
        for name, heads in (("q", hq), ("k", hkv), ("v", hkv)):
            state[name] = rand(b, s, heads, d).requires_grad_(train)
        for name in ("q_weight", "k_weight"):
            state[name] = (1.0 + 0.1 * rand(d)).requires_grad_(train)
        freq = 10000.0 ** (-torch.arange(0, d, 2, device=dev, dtype=torch.float32) / d)
        angle = torch.arange(s, device=dev, dtype=torch.float32)[:, None] * freq[None]
        angle = torch.cat([angle, angle], dim=-1)[None]
        state["cos"], state["sin"] = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
        state["d_o"] = rand(b, s, hq, d).transpose(1, 2)
        return state
    state["q"] = rand(b, hq, s, d).requires_grad_(train)
    state["k"] = rand(b, hkv, s, d).requires_grad_(train)
    state["v"] = rand(b, hkv, s, d).requires_grad_(train)
    state["d_o"] = rand(b, hq, s, d)
    state["segments"] = None
    if case["kind"] == "packed":
        ids, starts, _ = _case_segments(case, seed)
        state["segments"] = PackedMask(seg_id=ids.to(dev), seg_start=starts.to(dev))
    return state


def run(state):
    case = state["case"]
    train = case["step"] == "train"
    with torch.set_grad_enabled(train):
        if case["kind"] == "loss":
            hidden, head, targets = state["hidden"], state["head"], state["targets"]
            if not train:
                nll, lse, tgt = fused_linear_ce(hidden, head, targets)
                return {"nll": nll, "lse": lse, "target_logit": tgt}
            loss, count = reduced_linear_cross_entropy(hidden, head, targets)
            wanted = [hidden] + ([head.weight] if case["head"] == "trained" else [])
            grads = torch.autograd.grad(loss, wanted)
            return {"loss": loss.detach(), "count": count, "grads": list(grads)}
        q, k, v = state["q"], state["k"], state["v"]
        if case["kind"] == "layer":
            cos, sin, qw, kw = state["cos"], state["sin"], state["q_weight"], state["k_weight"]
            o = flash_attention(qk_norm_rope(q, cos, sin, weight=qw).transpose(1, 2),
                                qk_norm_rope(k, cos, sin, weight=kw).transpose(1, 2), v.transpose(1, 2),
                                scale=state["scale"])
            wanted = (q, k, v, qw, kw)
        else:
            o = flash_attention(q, k, v, scale=state["scale"], segments=state["segments"])
            wanted = (q, k, v)
        if not train:
            return {"o": o}
        return {"o": o.detach(), "grads": list(torch.autograd.grad(o, wanted, state["d_o"]))}


def work(case):
    """Bytes: every input once, every output once.  Flops: a loss needs the logits and, with gradients, one more
    contraction for each gradient; causal attention two products forward and five backward over half the square."""
    train = case["step"] == "train"
    if case["kind"] == "loss":
        n, d, v = case["n"], case["d"], case["v"]
        item = 4 if case["dtype"] == "fp32" else 2
        head = v * d * (0.5 + 4 / 64) if case["head"] == "int4" else v * d * item
        passes = 1 + train + (case["head"] == "trained")
        moved = n * d * item * (1 + train) + head * (1 + (case["head"] == "trained")) + 8 * n + 12 * n * (not train)
        return {"bytes": moved, "flops": 2.0 * passes * n * d * v}
    b, s, hq, hkv, d = (case[k] for k in ("b", "s", "hq", "hkv", "d"))
    q, kv = 2 * b * hq * s * d, 2 * b * hkv * s * d
    moved = 2 * q + 2 * kv + ((2 * q + 2 * kv) if train else 0)
    # packed documents: the mean square of a length uniform in [lo, hi] over its mean, times the row
    pairs = float(s) * s
    if case["kind"] == "packed":
        lo, hi = case["seg_lo"], min(case["seg_hi"], s)
        pairs = s * (lo * lo + lo * hi + hi * hi) / 3.0 / ((lo + hi) / 2.0)
    return {"bytes": moved, "flops": (7.0 if train else 2.0) * b * hq * pairs * d}


def tolerance(case):
    """About four times the distance to the same sums in float64: bf16 gradients and attention outputs 2.0e-3 to
    2.7e-3 (single values up to 5e-2 of the r.m.s. for losses, 9e-2 for attention), fp32 losses and gradients
    up to 1.5e-6, per-token losses of bf16 operands up to 4.3e-6."""
    if case["kind"] == "loss":
        if case["step"] == "eval":
            return {"rel": 1.7e-5, "max": 2e-4}
        if case["dtype"] == "fp32":
            return {"rel": 6e-6, "max": 2e-4}
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 1e-2, "max": 0.36}
