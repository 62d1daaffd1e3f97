"""Tensor-core attention backward (16-bit tensors, head_dim 32 / 64 / 128) at the edges of its 64-row tiles against torch
autograd of the fp32 masked softmax.

Tolerance: inputs are exact in both, P and dS enter their products with at least 16 significant bits and accumulate in fp32,
so a gradient is off by its own rounding (2^-9 of its value for bf16, 2^-12 for fp16), by the 16-bit rounding of the forward's output in
delta = rowsum(dO O) (which moves dS by P times 2^-9 |dO||O|) and by the approximate exp2 (2 ulp); 1e-2 (bf16) and 2e-3 (fp16) of the
largest gradient bound their sum.  How many bits P and dS keep shows in `test_gradients_of_any_size_keep_their_bits`."""
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


@pytest.mark.parametrize("dtype,size", [(torch.bfloat16, 1.0), (torch.bfloat16, 1e-6), (torch.float16, 1.0), (torch.float16, 2e4), (torch.float16, 1e-4),
                                        (torch.float16, 1e-6)])
@pytest.mark.parametrize("length,dim", [(40, 32), (130, 64), (300, 64), (200, 128)])
def test_gradients_of_any_size_keep_their_bits(length, dim, dtype, size):
    """Upstream gradients as loss scaling makes them and as small as fp16 holds them, against float64 for the same 16-bit output.

    Bound per element: the rounding of the result (half a unit: 2^-9 / 2^-12 of its value, 2^-25 where fp16 is subnormal; doubled)
    plus 2^-16 of the sum's absolute terms: 2^-18 for the two parts of P and dS, 2^-21 for two exp2 of 2 ulp, some 2^-18 for the fp32 sums
    of 32 to 128 terms in the scores and in dP.  One 16-bit part (2^-9, 2^-12) exceeds it, and so does a split that leaves fp16's range."""
    g = torch.Generator(device="cuda").manual_seed(length)
    batch, heads = 2, 3
    q, k, v, d_o = (torch.randn(batch, heads, length, dim, device="cuda", generator=g).to(dtype) for _ in range(4))
    d_o = (d_o.float().clamp(-3, 3) * size).to(dtype)
    lens = torch.tensor([length, length * 2 // 3], dtype=torch.int32, device="cuda")
    out = ops.varlen_attention(q, k, v, seq_len=lens, causal=True)
    got = ops.attention_backward(q, k, v, out, d_o, seq_len=lens, causal=True)
    qd, kd, vd, od, gd = (t.double() for t in (q, k, v, out, d_o))
    scale = dim ** -0.5
    pos = torch.arange(length, device="cuda")
    seen = (pos[None, :] <= pos[:, None])[None] & (pos[None, None, :] < lens[:, None, None])
    p = torch.softmax((qd @ kd.transpose(-1, -2) * scale).masked_fill(~seen[:, None], float("-inf")), -1)
    ds = p * (gd @ vd.transpose(-1, -2) - (gd * od).sum(-1, keepdim=True))
    ds_abs = p * (gd.abs() @ vd.abs().transpose(-1, -2) + (gd * od).abs().sum(-1, keepdim=True))
    unit = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    step = 2.0 ** -24 if dtype == torch.float16 else 0.0
    for name, x, want, terms in (("dq", got[0], ds @ kd * scale, ds_abs @ kd.abs() * scale),
                                 ("dk", got[1], ds.transpose(-1, -2) @ qd * scale, ds_abs.transpose(-1, -2) @ qd.abs() * scale),
                                 ("dv", got[2], p.transpose(-1, -2) @ gd, p.transpose(-1, -2) @ gd.abs())):
        fits = want.abs() < torch.finfo(dtype).max * 0.999
        err = (x.double() - want).abs()[fits]
        bound = (unit * want.abs() + step + 2.0 ** -16 * terms)[fits]
        assert bool((err <= bound).all()), f"{name}: {(err / bound.clamp_min(1e-300)).max().item():.2f} of the bound"
        assert bool((x[~fits].abs() > 0.99 * torch.finfo(dtype).max).all()), name
