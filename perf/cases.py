"""The work that is timed: what a user of this package has it do, through its public entry points.

Two groups of users.  Some score batches with the inference engine (``OneTransInference.scores`` on batches that are
on the GPU, ``score_stream`` on pinned host batches).  Others keep their own model and call the operators that stand
behind its norms, attention, embedding bags and FFN, in evaluation and in training.

``listed`` names twelve fixed cases and ``draw`` gives more of the same kinds: request-sized to full-scale batches, odd
sizes among them, 16-bit and 32-bit types, forward alone and forward with backward.  Model sizes, lengths, id
distributions and operator shapes are those of ``bench.py`` and of the tests.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from taac_2026_b200 import ops
from taac_2026_b200.inputs import EntityInput, ModelInput, OneTransSpec, SequenceInput, compact_model_input
from taac_2026_b200.onetrans import OneTransInference, pyramid_keep_count, random_state_dict, score_stream

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_ESIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
_NOW = 1_700_000_000  # request time of every sample


def listed() -> list[dict]:
    full = dict(d=512, heads=8, blocks=8, emb=128, fields=64, seq_vocab=1_000_000, buckets=0, id_exp=1.1)
    base = dict(d=128, heads=4, blocks=2, emb=64, fields=32, seq_vocab=1_000_000, buckets=0, id_exp=1.2)
    return [
        # one page request with a handful of candidates on the full-scale backbone: latency
        dict(name="score_request", kind="score", batch=8, length=1024, min_len=128, vocab=100_000, dtype="bf16", ffn="fp8", **full),
        # an evaluation batch of the reference's own size on the same backbone, with the engine's default FFN precision
        dict(name="score_batch", kind="score", batch=512, length=512, min_len=64, vocab=100_000, dtype="bf16", ffn="bf16", **full),
        # the full-scale configuration: one GPU's share of the global batch, 64 tables of a million rows
        dict(name="score_full", kind="score", batch=8192, length=1024, min_len=128, vocab=1_000_000, dtype="bf16", ffn="fp8", **full),
        # the baseline-sized model in the fp32 mode, for runs whose scores are compared with the reference's
        dict(name="score_base_fp32", kind="score", batch=512, length=256, min_len=16, vocab=100_000, dtype="fp32", ffn="bf16", **base),
        # the evaluation loop: pinned host batches in, scores out, copies included
        dict(name="score_stream", kind="stream", count=4, batch=2048, length=1024, min_len=128, vocab=100_000, dtype="bf16", ffn="fp8", **full),
        # the normalisation of a small model's tokens (the size of the reference's own operator benchmark)
        dict(name="rms_norm_small", kind="norm", op="rms", rows=8192, cols=128, dtype="fp16", train=False),
        # the widest rows of the normalisation sweep
        dict(name="layer_norm_wide", kind="norm", op="layer", rows=65_536, cols=1024, dtype="bf16", train=False),
        # a training step's normalisation, forward and backward
        dict(name="layer_norm_train", kind="norm", op="layer", rows=65_536, cols=512, dtype="bf16", train=True),
        # pooling of a multi-valued sparse field (the reference's operator benchmark)
        dict(name="bag_mean", kind="bag", batch=8192, bag=8, dim=128, vocab=1_000_000, dtype="fp16", train=False),
        # ragged behaviour sequences padded to one length, causal, lengths known to the caller
        dict(name="attention_ragged", kind="attention", form="lengths", batch=256, heads=8, length=1024, min_len=32, dim=64,
             causal=True, dtype="bf16", train=False),
        # the reference's models in training: attention with a bool mask [B, H, T, T], forward and backward
        dict(name="attention_train", kind="attention", form="mask", batch=64, heads=8, length=256, min_len=16, dim=64,
             causal=True, dtype="bf16", train=True),
        # the e4m3 SiLU-gated FFN over the tokens of a large batch
        dict(name="ffn_gated", kind="ffn", rows=262_144, d=512, hidden=2048, gated=True, mode="fp8"),
    ]


def _log(rng, low: int, high: int) -> int:
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng) -> dict:
    kind = rng.choice(["score", "score", "score", "stream", "norm", "norm", "bag", "attention", "attention", "ffn"])
    if kind in ("score", "stream"):
        d, heads = rng.choice([(128, 4), (128, 2), (256, 4), (512, 8), (512, 8)])
        fp32 = kind == "score" and d == 128 and rng.random() < 0.4
        length = 2 * _log(rng, 16, 512)
        case = dict(kind=kind, batch=_log(rng, 1, 1024 if fp32 else 8192), length=length, min_len=rng.randint(1, max(1, length // 8)),
                    vocab=_log(rng, 10_000, 300_000), dtype="fp32" if fp32 else "bf16",
                    ffn="bf16" if d == 128 else rng.choice(["bf16", "fp8", "fp8"]),
                    d=d, heads=heads, blocks=rng.randint(2, 8 if d == 512 else 4), emb=64 if d == 128 else 128,
                    fields=rng.randint(8, 64), seq_vocab=_log(rng, 100_000, 1_000_000), buckets=rng.choice([0, 65]),
                    id_exp=round(rng.uniform(1.05, 1.3), 3))
        if kind == "stream":
            case.update(count=rng.randint(2, 4), batch=_log(rng, 16, 2048))
        else:
            case["length"] -= rng.randint(0, 1)
        return case
    if kind == "norm":
        train = rng.random() < 0.4
        cols = rng.choice([128, 256, 512, 1024, 8 * rng.randint(8, 128), rng.randint(33, 1024)])
        if train:
            cols = max(64, cols // 8 * 8)
        return dict(kind="norm", op=rng.choice(["rms", "layer"]), rows=_log(rng, 64, 65_536), cols=cols,
                    dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]) if not train else "bf16", train=train)
    if kind == "bag":
        return dict(kind="bag", batch=_log(rng, 64, 16_384), bag=rng.randint(1, 12), dim=rng.choice([64, 128, 8 * rng.randint(4, 32)]),
                    vocab=_log(rng, 10_000, 1_000_000), dtype=rng.choice(["fp16", "bf16", "fp32"]), train=rng.random() < 0.3)
    if kind == "attention":
        train = rng.random() < 0.4
        form = "mask" if train else rng.choice(["lengths", "lengths", "mask", "none"])
        length = _log(rng, 17, 512 if train else 1024)
        heads, dim = rng.choice([(4, 32), (8, 64), (8, 64), (4, 64), (4, 128)])
        most = 64 * 8 * 256 * 256 if train else 256 * 8 * 1024 * 1024 // 4
        batch = _log(rng, 1, max(1, min(256, most // (heads * length * length))))
        return dict(kind="attention", form=form, batch=batch, heads=heads, length=length, min_len=rng.randint(1, max(1, length // 8)), dim=dim,
                    causal=rng.random() < 0.6, dtype=rng.choice(["bf16", "bf16", "fp16"]), train=train)
    return dict(kind="ffn", rows=_log(rng, 64, 262_144), d=rng.choice([256, 512]), hidden=rng.choice([1024, 2048]), gated=rng.random() < 0.5,
                mode=rng.choice(["fp8", "fp8", "mx", "precise"]))


# --------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------
def _zipf(shape, vocab: int, exponent: float, g: torch.Generator) -> torch.Tensor:
    """Ids in [1, vocab] with P(r) proportional to r ** -exponent; id 0 stays the padding id."""
    cdf = torch.cumsum(torch.arange(1, vocab + 1, dtype=torch.float64, device="cuda").pow_(-exponent), dim=0)
    u = torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=vocab - 1) + 1


def _spec(case: dict) -> OneTransSpec:
    users = case["fields"] * 3 // 4
    return OneTransSpec(
        user_int_specs=[(case["vocab"], i, 1) for i in range(users)],
        item_int_specs=[(case["vocab"], i, 1) for i in range(case["fields"] - users)],
        user_dense_dim=16, item_dense_dim=0, seq_vocab_sizes={"seq_a": [case["seq_vocab"]]}, d_model=case["d"], emb_dim=case["emb"],
        num_blocks=case["blocks"], num_heads=case["heads"], hidden_mult=4, seq_top_k=case["length"], num_time_buckets=case["buckets"],
        user_ns_tokens=5, item_ns_tokens=2)


def _record(case: dict, spec: OneTransSpec, g: torch.Generator) -> ModelInput:
    batch, length = case["batch"], case["length"]

    def entity(fields: int, dense: int) -> EntityInput:
        return EntityInput(_zipf((batch, fields), case["vocab"], case["id_exp"], g),
                           torch.rand(batch, fields, device="cuda", generator=g) < 0.02,
                           torch.randn(batch, dense, device="cuda", generator=g), torch.zeros(batch, dense, dtype=torch.bool, device="cuda"))

    lens = torch.randint(case["min_len"], length + 1, (batch,), device="cuda", generator=g)
    valid = torch.arange(length, device="cuda")[None, :] < lens[:, None]
    values = torch.where(valid, _zipf((batch, length), case["seq_vocab"], 1.1, g), 0)[:, None, :].contiguous()
    stamps = torch.zeros(batch, length, dtype=torch.int64, device="cuda")
    if case["buckets"]:  # events of the last weeks, the newest one last
        gaps = torch.randint(1, 3600, (batch, length), device="cuda", generator=g).flip(1).cumsum(1).flip(1)
        stamps = torch.where(valid, _NOW - gaps, 0)
    return ModelInput(entity(len(spec.user_int_specs), 16), entity(len(spec.item_int_specs), 0),
                      {"seq_a": SequenceInput(values, lens, stamps)}, torch.full((batch,), _NOW, dtype=torch.int64, device="cuda"))


def _mask(lens: torch.Tensor, length: int, causal: bool, heads: int) -> torch.Tensor:
    """The bool mask [B, H, T, T] that the models hand over: valid keys, and under ``causal`` no later ones, where
    a padded query sees itself alone."""
    pos = torch.arange(length, device="cuda")
    valid = pos[None, :] < lens[:, None]
    if not causal:
        return valid[:, None, None, :].expand(-1, heads, length, -1)
    mask = torch.where(valid[:, :, None], valid[:, None, :] & (pos[None, None, :] <= pos[None, :, None]), pos[None, None, :] == pos[None, :, None])
    return mask[:, None].expand(-1, heads, -1, -1)


def prepare(case: dict, seed: int):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("score", "stream"):
        spec, dtype = _spec(case), _DTYPES[case["dtype"]]
        weights = random_state_dict(spec, seed=seed + 1, device="cuda", dtype=dtype)
        model = OneTransInference(weights, spec, dtype=dtype, ffn=case["ffn"])
        if kind == "score":
            return {"case": case, "model": model, "batch": _record(case, spec, g)}
        host = []
        for _ in range(case["count"]):
            packed = compact_model_input(_record(case, spec, g).to("cpu"), threads=4)
            host.append(packed.pin_memory())
        return {"case": case, "model": model, "batches": host}
    dtype = _DTYPES[case.get("dtype", "bf16")]
    if kind == "norm":
        rows, cols, train = case["rows"], case["cols"], case["train"]
        x = torch.randn(rows, cols, device="cuda", generator=g)
        x[torch.rand(rows, device="cuda", generator=g) < 0.01] *= 50.0
        state = {"case": case, "x": x.to(dtype), "w": (1 + 0.02 * torch.randn(cols, device="cuda", generator=g)).to(dtype),
                 "b": (0.02 * torch.randn(cols, device="cuda", generator=g)).to(dtype)}
        if train:
            for name in ("x", "w", "b"):
                state[name].requires_grad_()
            state["grad"] = torch.randn(rows, cols, device="cuda", generator=g).to(dtype)
        return state
    if kind == "bag":
        ids = torch.randint(1, case["vocab"], (case["batch"], case["bag"]), device="cuda", generator=g)
        ids[torch.rand(ids.shape, device="cuda", generator=g) < 0.25] = 0
        table = torch.randn(case["vocab"], case["dim"], device="cuda", generator=g).to(dtype)
        table[0] = 0
        return {"case": case, "table": table, "ids": ids,
                "grad": torch.randn(case["batch"], case["dim"], device="cuda", generator=g).to(dtype)}
    if kind == "attention":
        batch, heads, length, dim = case["batch"], case["heads"], case["length"], case["dim"]
        q, k, v, grad = (torch.randn(batch, heads, length, dim, device="cuda", generator=g).to(dtype) for _ in range(4))
        lens = torch.randint(case["min_len"], length + 1, (batch,), device="cuda", generator=g)
        state = {"case": case, "q": q, "k": k, "v": v, "lens": lens.to(torch.int32)}
        if case["form"] == "mask":
            state["mask"] = _mask(lens, length, case["causal"], heads)
        if case["train"]:
            state["grad"] = grad
            for t in (q, k, v):
                t.requires_grad_()
        return state
    d, hidden = case["d"], case["hidden"]
    t4 = torch.randn(case["rows"], d, device="cuda", generator=g)
    tail = torch.rand(case["rows"], 1, device="cuda", generator=g) < 0.01  # rows with outliers
    x = torch.where(tail, t4 * 8.0, t4).to(torch.bfloat16)
    w_up = (0.02 * torch.randn((2 if case["gated"] else 1) * hidden, d, device="cuda", generator=g)).to(torch.bfloat16)
    w_down = (0.02 * torch.randn(d, hidden, device="cuda", generator=g)).to(torch.bfloat16)
    make = ops.MxFfnWeights if case["mode"] == "mx" else ops.Fp8FfnWeights
    more = {"precise": True} if case["mode"] == "precise" else {}
    return {"case": case, "x": x, "weights": make(w_up, w_down, gated=case["gated"], **more)}


# --------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "score":
        return state["model"].scores(state["batch"])
    if kind == "stream":
        return list(score_stream(state["model"], state["batches"]))
    if kind == "norm":
        x, w, b = state["x"], state["w"], state["b"]
        if case["op"] == "rms":
            y = ops.rms_norm(x, w)
            return y if not case["train"] else (y.detach(), *torch.autograd.grad(y, (x, w), state["grad"]))
        y = ops.layer_norm(x, w, b)
        return y if not case["train"] else (y.detach(), *torch.autograd.grad(y, (x, w, b), state["grad"]))
    if kind == "bag":
        out = ops.embedding_bag_mean(state["table"], state["ids"])
        if not case["train"]:
            return out
        grad = ops.embedding_bag_mean_backward(state["ids"], state["grad"], case["vocab"])
        return out, grad._indices(), grad._values()
    if kind == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        if case["form"] == "lengths":
            return ops.varlen_attention(q, k, v, seq_len=state["lens"], causal=case["causal"])
        out = ops.flash_attention(q, k, v, attn_mask=state.get("mask"), is_causal=case["causal"] and case["form"] == "none")
        return out if not case["train"] else (out.detach(), *torch.autograd.grad(out, (q, k, v), state["grad"]))
    if case["mode"] == "mx":
        return ops.ffn_mx(state["x"], state["weights"])
    return ops.ffn_fp8(state["x"], state["weights"], precise=case["mode"] == "precise")


# --------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two right answers may differ
# --------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _distinct(vocab: int, length: int) -> float:
    """Distinct ids among ``length`` draws of the sequence distribution."""
    p = np.arange(1, vocab + 1, dtype=np.float64) ** -1.1
    return float(-np.expm1(length * np.log1p(-p / p.sum())).sum())


def _score_work(case: dict) -> dict:
    """Tokens by the mean of the length distribution, an event counted once per sample.  Every layer projects keys and values of
    its rows and runs the rest for the rows that the pyramid hands on; the non-sequence tokens have weights of their own."""
    batch, d, blocks, length, emb, es = case["batch"], case["d"], case["blocks"], case["length"], case["emb"], _ESIZE[case["dtype"]]
    ns, fields = 9, case["fields"]  # 5 + 2 sparse tokens, one dense, one of sequence statistics
    low, steps = case["min_len"], 16
    lens = [_distinct(case["seq_vocab"], round(low + (length - low) * (i + 0.5) / steps)) for i in range(steps)]
    mean = sum(lens) / steps
    flops = 2 * batch * (mean * emb * d + fields * emb * 5 * d + 2 * d * d)
    width, dropped = length, 0
    for layer in range(blocks):
        keep = pyramid_keep_count(width, layer, blocks, ns)
        now = [max(0.0, n - dropped) for n in lens]
        dropped += width - keep
        after = [max(0.0, n - dropped) for n in lens]
        rows, kept = sum(now) / steps + ns, sum(after) / steps + ns
        pairs = sum((a + ns) * ((n + ns) - (a + ns) / 2) for n, a in zip(now, after)) / steps
        flops += batch * (4 * rows * d * d + kept * (4 + 16) * d * d + 4 * pairs * d)
        width = keep
    weights = blocks * (d * d * (3 + 1 + 8) + ns * d * d * (3 + 8)) + fields * emb * 5 * d + emb * d + 2 * d * d
    bytes_ = weights * es + batch * (fields * (8 + 1 + emb * es) + length * 8 * (2 if case["buckets"] else 1) + mean * emb * es + 100)
    return {"bytes": bytes_, "flops": flops}


def _pairs(case: dict) -> float:
    length, low = case["length"], case["min_len"]
    if case["form"] == "none":
        lens = [float(length)]
    else:
        lens = [low + (length - low) * (i + 0.5) / 64 for i in range(64)]
    return case["batch"] * case["heads"] * sum(n * n / 2 if case["causal"] else n * n for n in lens) / len(lens)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "score":
        return _score_work(case)
    if kind == "stream":
        one = _score_work(case)
        return {"bytes": case["count"] * one["bytes"], "flops": case["count"] * one["flops"]}
    if kind == "norm":
        size = case["rows"] * case["cols"] * _ESIZE[case["dtype"]]
        return {"bytes": size * (5 if case["train"] else 2), "flops": case["rows"] * case["cols"] * (16 if case["train"] else 6)}
    if kind == "bag":
        batch, bag, dim, es = case["batch"], case["bag"], case["dim"], _ESIZE[case["dtype"]]
        bytes_ = batch * (8 * bag + 0.75 * bag * dim * es + dim * es)
        if case["train"]:
            bytes_ += batch * (8 * bag + dim * es + bag * (8 + dim * es))
        return {"bytes": bytes_, "flops": batch * bag * dim}
    if kind == "attention":
        size = case["batch"] * case["heads"] * case["length"] * case["dim"] * 2
        flops = 4 * case["dim"] * _pairs(case)
        bytes_ = 4 * size + (case["batch"] * case["length"] ** 2 if case["form"] == "mask" and case["causal"] else 0)
        if case["train"]:
            bytes_, flops = bytes_ + 8 * size, 3.5 * flops
        return {"bytes": bytes_, "flops": flops}
    rows, d, hidden = case["rows"], case["d"], case["hidden"]
    weights = (3 if case["gated"] else 2) * d * hidden
    return {"bytes": rows * d * 4 + weights, "flops": 2 * rows * weights}


def tolerance(case: dict) -> dict:
    kind, dtype = case["kind"], case.get("dtype", "bf16")
    if kind in ("score", "stream"):
        # scores lie around one half; a 16-bit network moves them by some 1e-4 to 5e-4
        return {"rel": 1e-5} if dtype == "fp32" else {"rel": 2e-3, "max": 1e-2}
    if kind == "ffn":
        return {"rel": 1e-2}
    if dtype == "fp32":
        return {"rel": 1e-5}
    if kind == "bag":
        return {"rel": 1e-3 if dtype == "fp16" else 5e-3}
    if kind == "norm":
        return {"rel": 1e-3 if dtype == "fp16" else 1e-2}
    return {"rel": 3e-3 if dtype == "fp16" else 1e-2}
