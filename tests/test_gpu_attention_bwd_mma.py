"""Tensor-core attention backward (16-bit tensors, head_dim 32 / 64 / 128) at the edges of its 64-row tiles against torch
autograd of the fp32 masked softmax.

Tolerance: inputs are exact in both, P and dS enter their products with at least 16 significant bits and accumulate in fp32,
so a gradient is off by its own rounding (2^-9 of its value for bf16, 2^-12 for fp16), by the 16-bit rounding of the forward's output in
delta = rowsum(dO O) (which moves dS by P times 2^-9 |dO||O|) and by the approximate exp2 (2 ulp); 1e-2 (bf16) and 2e-3 (fp16) of the
largest gradient bound their sum."""
from __future__ import annotations

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200 import ops
from test_gpu_attention_bwd import _mask, _reference

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("lq,lk,dim,causal,ns,padded_self,key_map", [
    (64, 64, 64, True, 0, False, False), (65, 65, 64, True, 9, True, False), (63, 63, 32, False, 0, False, False),
    (128, 200, 64, False, 5, False, False), (193, 193, 128, True, 3, True, False), (1, 1, 64, True, 0, False, False),
    (130, 130, 32, True, 0, True, True), (129, 257, 128, False, 0, False, False), (300, 300, 64, True, 0, True, False),
])
def test_backward_at_tile_edges(lq, lk, dim, causal, ns, padded_self, key_map, dtype, tol):
    g = torch.Generator().manual_seed(lq * 31 + dim)
    batch, heads = 3, 2
    q, k, v = (torch.randn(batch, heads, n, dim, generator=g).to(dtype) for n in (lq, lk, lk))
    grad = torch.randn(batch, heads, lq, dim, generator=g).to(dtype)
    ns_start = lk - ns
    lens = torch.randint(0, ns_start + 1, (batch,), generator=g)
    lens[0] = 0
    valid = None
    if key_map:
        valid = torch.rand(batch, lk, generator=g) < 0.6
    visible = _mask(batch, lq, lk, lens, ns_start, causal, padded_self, key_valid=valid)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    _reference(qr, kr, vr, visible, dim ** -0.5).backward(grad.float())
    mask = dict(causal=causal, padded_query_self=padded_self)
    mask.update(dict(key_valid=valid.cuda()) if key_map else dict(seq_len=lens.to(torch.int32).cuda(), ns_start=ns_start))
    out = ops.varlen_attention(q.cuda(), k.cuda(), v.cuda(), layout="bhld", **mask)
    got = ops.attention_backward(q.cuda(), k.cuda(), v.cuda(), out, grad.cuda(), **mask)
    for name, x, want in zip(("dq", "dk", "dv"), got, (qr.grad, kr.grad, vr.grad)):
        err = (x.float().cpu() - want).abs().max().item()
        assert err <= tol * max(1.0, want.abs().max().item()), f"{name}: {err}"
