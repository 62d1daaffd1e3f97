"""Weights that change under a model that has scored already, and first calls on several streams: scores are those of a model
built from the present weights.  The forward keeps casts, transposes and three-part splits of weights; none of them may outlive the
tensor, or the content, it was made from."""
from __future__ import annotations

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200.inputs import EntityInput, ModelInput, OneTransSpec, SequenceInput
from taac_2026_b200.onetrans import OneTransInference, random_state_dict

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


def _spec(d=128, heads=4, dense=4):
    return OneTransSpec(user_int_specs=[(50, i, 1) for i in range(4)], item_int_specs=[(50, i, 1) for i in range(3)], user_dense_dim=dense, item_dense_dim=0,
                        seq_vocab_sizes={"seq_a": [100]}, d_model=d, emb_dim=64, num_blocks=2, num_heads=heads, hidden_mult=4, seq_top_k=32,
                        num_time_buckets=0, user_ns_tokens=3, item_ns_tokens=2)


def _batch(batch=11, length=24, dense=4, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ids = lambda *s, high: torch.randint(1, high, s, device="cuda", generator=g)  # noqa: E731

    def entity(fields, width):
        return EntityInput(ids(batch, fields, high=50), torch.zeros(batch, fields, dtype=torch.bool, device="cuda"),
                           torch.randn(batch, width, device="cuda", generator=g), torch.zeros(batch, width, dtype=torch.bool, device="cuda"))

    lens = torch.randint(1, length + 1, (batch,), device="cuda", generator=g)
    values = torch.where(torch.arange(length, device="cuda")[None] < lens[:, None], ids(batch, length, high=100), 0)[:, None].contiguous()
    zeros = torch.zeros(batch, length, dtype=torch.int64, device="cuda")
    return ModelInput(entity(4, dense), entity(3, 0), {"seq_a": SequenceInput(values, lens, zeros)}, torch.full((batch,), 10, dtype=torch.int64, device="cuda"))


def _model(spec, weights, dtype, ffn="bf16"):
    return OneTransInference({k: v.clone() for k, v in weights.items()}, spec, dtype=dtype, ffn=ffn)


@pytest.mark.parametrize("dtype,d,ffn", [(torch.float32, 128, "bf16"), (torch.bfloat16, 128, "bf16"), (torch.bfloat16, 256, "bf16"), (torch.bfloat16, 256, "fp8")])
def test_replaced_block_entries_are_read(dtype, d, ffn):
    spec, batch = _spec(d), _batch()
    weights, others = (random_state_dict(spec, seed=s, device="cuda", dtype=dtype) for s in (1, 2))
    model = _model(spec, weights, dtype, ffn)
    first = model.scores(batch).clone()
    changed = {k: (others[k] if ".attention.shared_qkv.weight" in k or ".ffn.shared." in k else v) for k, v in weights.items()}
    want = _model(spec, changed, dtype, ffn)
    for blk, new in zip(model.blocks, want.blocks):       # the same keys, the same number of entries
        for key in ("qkv_w", "q_w", "kv_w", "ffn_w1", "ffn_b1", "ffn_w2", "ffn_b2", "ffn_fp8", "ffn_fp8_folded"):
            if key in blk:
                blk[key] = new[key]
    expected = want.scores(batch)
    assert not torch.equal(expected, first)
    assert torch.equal(model.scores(batch), expected)
    model.blocks = _model(spec, weights, dtype, ffn).blocks
    assert torch.equal(model.scores(batch), first)


def test_replaced_ffn_attributes_are_read():
    spec, batch = _spec(256), _batch()
    model = _model(spec, random_state_dict(spec, seed=1, device="cuda", dtype=torch.bfloat16), torch.bfloat16, "fp8")
    first = model.scores(batch).clone()
    for blk in model.blocks:
        blk["ffn_fp8_folded"].b_down = blk["ffn_fp8_folded"].b_down + 1.0
    assert not torch.equal(model.scores(batch), first)


@pytest.mark.parametrize("name", ["blocks.0.attention.out.weight", "blocks.1.attention.shared_qkv.weight", "blocks.0.ffn.shared.net.0.weight",
                                  "classifier.0.weight", "classifier.3.weight", "classifier.3.bias", "sequence_stats_projector.0.weight",
                                  "user_dense.project.0.weight", "user_dense.project.2.bias", "user_tokenizer.project.0.weight",
                                  "sequence_tokenizers.seq_a.project.0.weight"])
def test_fp32_weights_changed_in_place_are_read(name):
    spec, batch = _spec(), _batch()
    weights = random_state_dict(spec, seed=3, device="cuda", dtype=torch.float32)
    model = _model(spec, weights, torch.float32)
    first = model.scores(batch).clone()
    with torch.no_grad():
        model.w[name].add_(0.25)
    expected = _model(spec, model.w, torch.float32).scores(batch)
    assert not torch.equal(expected, first)
    assert torch.equal(model.scores(batch), expected)


@pytest.mark.parametrize("name", ["classifier.3.bias", "sequence_stats_projector.2.weight"])
def test_weights_replaced_by_name_are_read(name):
    spec, batch = _spec(256), _batch()
    weights = random_state_dict(spec, seed=4, device="cuda", dtype=torch.bfloat16)
    model = _model(spec, weights, torch.bfloat16)
    first = model.scores(batch).clone()
    model.w[name] = model.w[name] * 3 + 1
    expected = _model(spec, model.w, torch.bfloat16).scores(batch)
    assert not torch.equal(expected, first)
    assert torch.equal(model.scores(batch), expected)


@pytest.mark.parametrize("order", ["prepare", "scores"])
def test_first_calls_on_two_streams(order):
    """The first call enqueues the splits of the weights behind 20 ms of other work on its stream; a call on another stream has to wait
    for them."""
    spec, batch = _spec(), _batch()
    weights = random_state_dict(spec, seed=5, device="cuda", dtype=torch.float32)
    expected = _model(spec, weights, torch.float32).scores(batch).clone()
    for _ in range(3):
        model = _model(spec, weights, torch.float32)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(40_000_000)
            if order == "prepare":
                model.prepare(batch)                              # converts what lies outside the blocks
            else:
                model._executor().load_blocks(model.blocks)       # and the blocks
        got = model.scores(batch)
        torch.cuda.synchronize()
        assert torch.equal(got, expected)


def test_a_dropped_result_keeps_its_landing_buffer():
    """The plan kernel of a prepared batch waits behind 20 ms of other work and writes pinned memory; the engine and the result are gone by
    then.  Pinned tensors that are made in between keep their values."""
    spec, batch = _spec(), _batch()
    model = _model(spec, random_state_dict(spec, seed=6, device="cuda", dtype=torch.bfloat16), torch.bfloat16)
    model.scores(batch)
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)
    for _ in range(4):                      # every buffer of the ring
        model.prepare(batch)
    model._native = None
    taken = [torch.full((2 * (spec.num_blocks + 1),), -7, dtype=torch.int64).pin_memory() for _ in range(16)]
    torch.cuda.synchronize()
    assert all(bool((t == -7).all()) for t in taken)
