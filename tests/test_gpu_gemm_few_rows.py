"""The GEMM forms for few rows per group at the edges of their dispatch (8, 16, 32, 128 rows) and of their tiles, against fp32 products
of the same bf16 operands.  Sums of K products in fp32 in another order differ by some 1e-6 of their terms; the result is rounded to bf16
(2^-9 of its value) and the tanh-form SiLU adds 2^-11: 1e-2 of the value plus 1e-2 of the scale bounds both (as for the large tiles)."""
from __future__ import annotations

import ctypes

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


def _close(got, want):
    return bool(((got.float() - want).abs() <= 1e-2 * want.abs() + 1e-2).all())


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 32, 33, 64, 100, 128, 129])
@pytest.mark.parametrize("groups,n,k", [(1, 256, 64), (9, 512, 512), (3, 256, 2048), (13, 1536, 192)])
def test_rows_around_the_dispatch_lines(m, groups, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    x = torch.randn(groups, m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(groups, n, k, device="cuda", generator=g) * k ** -0.5).bfloat16()
    b = torch.randn(groups, n, device="cuda", generator=g)
    r = torch.randn(groups, m, n, device="cuda", generator=g).bfloat16()
    ref = torch.einsum("gmk,gnk->gmn", x.float(), w.float()) + b[:, None]
    assert _close(ops.grouped_linear(x, w, b, silu=True, check=True), torch.nn.functional.silu(ref))
    want = ref + r.float()
    out = ops.grouped_linear(x, w, b, residual=r, out=r, check=True)              # in place on the residual
    assert out.data_ptr() == r.data_ptr() and _close(out, want)
    if m <= 64:                                                                   # gated: [128 gate | 128 value] rows
        gate, value = (t.reshape(groups, m, -1) for t in ref.view(groups, m, n // 256, 2, 128).unbind(3))
        assert _close(ops.grouped_linear(x, w, b, gated=True, check=True), torch.nn.functional.silu(gate) * value)


@pytest.mark.parametrize("m", [1, 8, 13, 32])
@pytest.mark.parametrize("biased", [False, True])
def test_norm_and_shared_weight(m, biased):
    groups, n, k = 3, 256, 512
    g = torch.Generator(device="cuda").manual_seed(m)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, w, b, gamma, nb = rand(groups, m, k).bfloat16(), (rand(n, k) * k ** -0.5).bfloat16(), rand(n), rand(k).bfloat16(), rand(k).bfloat16()
    out = torch.empty(groups, m, n, dtype=torch.bfloat16, device="cuda")
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
    code = _lib.load().tb200_gemm_bf16_few_rows(p(x), p(w), p(b), None, p(out), groups, m, n, k, 0, 1, p(gamma), p(nb if biased else None), 1e-6, None)
    assert code == 0
    normed = ops.rms_norm(x, gamma, 1e-6, in_bias=nb if biased else None)
    torch.cuda.synchronize()
    assert _close(out, normed.float() @ w.float().t() + b)


@pytest.mark.parametrize("batch,heads", [(3, 8), (300, 8)])                       # keys split over warps / one warp per (sample, head)
def test_last_rows_attention(batch, heads):
    g = torch.Generator(device="cuda").manual_seed(batch)
    n_q = 9
    lens = torch.randint(n_q, 150, (batch,), generator=g, device="cuda")
    cu = torch.zeros(batch + 1, dtype=torch.int32, device="cuda")
    cu[1:] = torch.cumsum(lens, 0)
    kv = torch.randn(int(cu[-1]), 2, heads, 64, device="cuda", generator=g).bfloat16()
    q = torch.randn(n_q, batch, heads, 64, device="cuda", generator=g).bfloat16()                 # token-major
    out = torch.empty_like(q)
    d = heads * 64
    st = (ctypes.c_int64 * 12)(d, 64, batch * d, 0, 64, 2 * d, 0, 64, 2 * d, d, 64, batch * d)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    code = _lib.load().tb200_attn_last_rows_fwd(p(q), p(kv), ctypes.c_void_p(kv.data_ptr() + 2 * d), p(out), batch, heads, n_q, 150, st, p(cu), 0.125,
                                                _lib.BF16, None)
    assert code == 0
    torch.cuda.synchronize()
    for b in range(0, batch, 37):
        lo, hi = int(cu[b]), int(cu[b + 1])
        s = torch.einsum("qhd,khd->hqk", q[:, b].float(), kv[lo:hi, 0].float()) * 0.125
        pos = torch.arange(hi - lo, device="cuda")
        s = s.masked_fill(pos[None, None] > (hi - lo - n_q + torch.arange(n_q, device="cuda"))[None, :, None], float("-inf"))
        want = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), kv[lo:hi, 1].float())
        assert (out[:, b].float() - want).abs().max().item() <= 2e-2
