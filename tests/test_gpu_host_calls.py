"""The host module's mask recognition (one kernel over the mask) against the tensor-arithmetic planner, at row widths around
its 16-byte pieces, and the refusal of masks that neither recognises."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import gpu_ready
from oracle import reference_ops as R
from taac_2026_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


def _qkv(batch, heads, length, seed):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(batch, heads, length, 64, generator=g).bfloat16().cuda() for _ in range(3))


@pytest.mark.parametrize("length", [1, 2, 15, 16, 17, 33, 64, 130, 265])
@pytest.mark.parametrize("form", ["key", "causal", "causal_ns", "full", "identity"])
def test_recognised_masks_give_the_planned_attention(length, form):
    batch, heads = 5, 2
    q, k, v = _qkv(batch, heads, length, length)
    ns = min(9, length - 1) if form == "causal_ns" else 0
    g = torch.Generator().manual_seed(length + 1)
    lens = torch.randint(0, length - ns + 1, (batch,), generator=g)
    if form == "full":
        lens[:] = length
    if form == "identity":
        lens[:] = 0
    causal = form != "key"
    mask = R.structured_attention_mask(lens, length, length - ns, causal, causal)[:, None].cuda()
    for m in (mask.expand(-1, heads, -1, -1), mask.repeat(1, heads, 1, 1)):
        plan = ops.plan_attention_mask(q, k, m, is_causal=False)
        want = ops.varlen_attention(q, k, v, seq_len=plan.seq_len, ns_start=plan.ns_start, causal=plan.causal,
                                    padded_query_self=plan.padded_query_self)
        assert ops._host.flash_attention(q, k, v, m, False) is not None      # not left to the tensor-arithmetic planner
        assert torch.equal(ops.flash_attention(q, k, v, attn_mask=m), want)


@pytest.mark.parametrize("flip", [(0, 0, 20), (3, 40, 40), (1, 64, 2), (4, 30, 31)])
def test_one_wrong_element_is_refused(flip):
    batch, heads, length = 5, 2, 65
    q, k, v = _qkv(batch, heads, length, 3)
    mask = R.structured_attention_mask(torch.tensor([65, 50, 30, 41, 9]), length, length, True, True)[:, None].clone().cuda()
    b, i, j = flip
    mask[b, 0, i, j] ^= True
    with pytest.raises(RuntimeError, match="cuda flash_attention"):
        ops.flash_attention(q, k, v, attn_mask=mask.expand(-1, heads, -1, -1))


@pytest.mark.parametrize("flag", [1, True, np.bool_(True)])
def test_flags_are_read_as_python_reads_them(flag):
    x, w, b = torch.randn(33, 64, device="cuda"), torch.rand(64, device="cuda"), torch.rand(64, device="cuda")
    want = torch.nn.functional.layer_norm(torch.nn.functional.silu(x), (64,), w, b, 1e-5)
    torch.testing.assert_close(ops.layer_norm(x, w, b, pre_silu=flag), want, atol=1e-5, rtol=1e-5)
    q, k, v = (torch.randn(2, 2, 20, 64, device="cuda").bfloat16() for _ in range(3))
    assert torch.equal(ops.varlen_attention(q, k, v, causal=flag), ops.varlen_attention(q, k, v, causal=True))


@pytest.mark.parametrize("make,call,name", [(ops.Fp8FfnWeights, ops.ffn_fp8, "s"), (ops.MxFfnWeights, ops.ffn_mx, "a")])
def test_ffn_scales_of_another_shape_are_refused(make, call, name):
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(40, 256, device="cuda", generator=g).bfloat16()
    w = [(0.05 * torch.randn(*s, device="cuda", generator=g)).bfloat16() for s in ((512, 256), (256, 512))]
    weights = make(*w, gated=False)
    want = call(x, weights).clone()
    for attr in (name + "_up", name + "_down"):
        whole = getattr(weights, attr)
        for wrong in (whole[:-1].contiguous(), whole[:, :1].contiguous()):
            setattr(weights, attr, wrong)
            with pytest.raises(ValueError):
                call(x, weights)
        setattr(weights, attr, whole)
    assert torch.equal(call(x, weights), want)


def test_whole_numbers_may_come_as_floats():
    q, k, v = (torch.randn(2, 2, 40, 64, device="cuda").bfloat16() for _ in range(3))
    lens = torch.tensor([12, 30], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.varlen_attention(q, k, v, seq_len=lens, ns_start=36.0), ops.varlen_attention(q, k, v, seq_len=lens, ns_start=36))
    ids = torch.randint(0, 50, (9, 4), device="cuda")
    assert ops.embedding_bag_mean_backward(ids, torch.ones(9, 64, device="cuda"), 50.0).shape == (50, 64)
