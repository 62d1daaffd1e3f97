"""Row kernels around the engine's blocks against plain fp32 tensor arithmetic, at the edges of their eight-row CTAs and with
widths that do not fill a warp.  fp32 sums of at most 2048 terms in another order differ by some 1e-6; results stored as bf16 by half a
unit in the last place, 2^-8 of the value between neighbours."""
from __future__ import annotations

import ctypes

import pytest
import torch
import torch.nn.functional as F

from conftest import gpu_ready
from taac_2026_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _code(dtype):
    return {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}[dtype]


def _tol(dtype):
    return dict(atol=2e-5, rtol=2e-5) if dtype == torch.float32 else dict(atol=2 ** -8, rtol=2 ** -8)


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,d,masked", [(1, 6, 64, False), (7, 16, 512, True), (9, 3, 96, True), (33, 6, 1024, False)])
def test_small_token(rows, n, d, masked, dtype):
    g = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    values, w, b, gamma, beta = rand(rows, n), rand(d, n * (1 + masked)) * 0.3, rand(d), rand(d), rand(d)
    mask = (rand(rows, n + 1) > 0) if masked else None
    x = torch.cat([values, mask[:, :n].float()], 1) if masked else values
    want = F.layer_norm(F.silu(F.linear(x, w, b)), (d,), gamma, beta)
    out = torch.full((rows, 2 * d), 7.0, dtype=dtype, device="cuda")
    code = _lib.load().tb200_small_token_fwd(_p(values), n, n, _p(mask), n + 1, w.shape[1], _p(w.t().contiguous()), _p(b), _p(gamma), _p(beta), _p(out), 2 * d, rows, d,
                                             1e-5, _code(dtype), None)
    assert code == 0
    torch.cuda.synchronize()
    torch.testing.assert_close(out[:, :d].float(), want, **_tol(dtype))
    assert bool((out[:, d:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,ns,d", [(1, 9, 64), (5, 9, 512), (13, 3, 264)])
def test_ns_rows_and_pooled_means(batch, ns, d, dtype):
    g = torch.Generator(device="cuda").manual_seed(d)
    lens = torch.randint(0, 5, (batch,), device="cuda", generator=g)
    cu = torch.zeros(batch + 1, dtype=torch.int64, device="cuda")
    cu[1:] = torch.cumsum(lens + ns, 0)
    total = int(cu[-1])
    ids = (cu[:-1] + lens)[None, :] + torch.arange(ns, device="cuda")[:, None]                     # token-major [ns, B]
    src = torch.randn(batch, ns, d, device="cuda", generator=g).to(dtype)
    w = torch.rand(d, device="cuda", generator=g).to(dtype)
    tokens = torch.randn(total, d, device="cuda", generator=g).to(dtype)
    normed, major = tokens.clone(), torch.empty(ns, batch, d, dtype=dtype, device="cuda")
    want = tokens.clone()
    want[ids.t().reshape(-1)] = src.view(-1, d)
    lib = _lib.load()
    assert lib.tb200_ns_rows_fwd(_p(src), batch, ns, d, _p(w), 1e-6, _p(ids), _p(tokens), _p(ids), _p(normed), _p(major), _code(dtype), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(tokens, want)
    torch.testing.assert_close(major.float(), _rms(src.float(), w.float()).transpose(0, 1), **_tol(dtype))
    assert torch.equal(normed[ids.reshape(-1)], major.view(-1, d))

    seq, mean = torch.empty(batch, d, device="cuda"), torch.empty(batch, d, device="cuda")
    assert lib.tb200_pool_rows_fwd(_p(tokens), _p(cu), _p(lens), batch, ns, d, _p(w), 1e-6, _p(seq), _p(mean), _code(dtype), None) == 0
    torch.cuda.synchronize()
    rows = _rms(tokens.float(), w.float())
    for b in range(batch):
        lo, n = int(cu[b]), int(lens[b])
        torch.testing.assert_close(seq[b], rows[lo:lo + n].mean(0) if n else torch.zeros(d, device="cuda"), atol=1e-5, rtol=1e-5)
        torch.testing.assert_close(mean[b], rows[lo + n:lo + n + ns].mean(0), atol=1e-5, rtol=1e-5)
    again = torch.empty(batch, d, device="cuda")
    assert lib.tb200_pool_rows_fwd(_p(tokens[ids.reshape(-1)].contiguous()), None, None, batch, ns, d, _p(w), 1e-6, None, _p(again), _code(dtype), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(again, mean)


@pytest.mark.parametrize("batch,d,actions", [(1, 64, 1), (9, 512, 3)])
def test_join_and_head(batch, d, actions):
    g = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    seq, ns, w, b = rand(batch, d), rand(batch, d), rand(actions, d) * 0.1, rand(actions)
    joined, cast = torch.empty(batch, 2 * d, device="cuda"), torch.empty(batch, 2 * d, dtype=torch.bfloat16, device="cuda")
    lib = _lib.load()
    assert lib.tb200_join_summaries(_p(seq), _p(ns), _p(joined), _p(cast), batch, d, _lib.BF16, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(joined, torch.cat([seq, ns], 1)) and torch.equal(cast, joined.bfloat16())
    assert lib.tb200_join_summaries(None, _p(ns), _p(joined), None, batch, d, _lib.BF16, None) == 0
    logits, probs = torch.empty(batch, actions, device="cuda"), torch.empty(batch, actions, device="cuda")
    h = rand(batch, d).bfloat16()
    assert lib.tb200_head_fwd(_p(h), _p(w), _p(b), _p(logits), _p(probs), batch, d, actions, _lib.BF16, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(joined, torch.cat([torch.zeros_like(ns), ns], 1))
    want = h.float() @ w.t() + b
    torch.testing.assert_close(logits, want, atol=2e-5, rtol=2e-5)
    torch.testing.assert_close(probs, torch.sigmoid(want), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ns,d", [(9, 64), (4, 264), (1, 512), (3, 1024)])
def test_pooled_means_of_many_samples(ns, d, dtype):
    """More than eight samples per SM: one warp per sample, rows four at a time and the remainder."""
    batch = 8 * torch.cuda.get_device_properties(0).multi_processor_count + 5
    g = torch.Generator(device="cuda").manual_seed(d)
    lens = torch.randint(0, 11, (batch,), device="cuda", generator=g)
    cu = torch.zeros(batch + 1, dtype=torch.int64, device="cuda")
    cu[1:] = torch.cumsum(lens + ns, 0)
    total = int(cu[-1])
    tokens = torch.randn(total, d, device="cuda", generator=g).to(dtype)
    w = torch.rand(d, device="cuda", generator=g).to(dtype)
    seq = torch.empty(batch * d + 1, device="cuda")[1:].view(batch, d)   # off a 16-byte boundary
    mean = torch.empty(batch, d, device="cuda")
    assert _lib.load().tb200_pool_rows_fwd(_p(tokens), _p(cu), _p(lens), batch, ns, d, _p(w), 1e-6, _p(seq), _p(mean), _code(dtype), None) == 0
    torch.cuda.synchronize()
    owner = torch.repeat_interleave(torch.arange(batch, device="cuda"), lens + ns)
    is_seq = torch.arange(total, device="cuda") - cu[:-1][owner] < lens[owner]
    rows = _rms(tokens.double(), w.double())
    for mask, count, got in ((is_seq, lens.clamp_min(1), seq), (~is_seq, torch.full_like(lens, ns), mean)):
        want = torch.zeros(batch, d, dtype=torch.float64, device="cuda").index_add_(0, owner[mask], rows[mask]) / count[:, None]
        torch.testing.assert_close(got.double(), want, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("batch,d", [(3, 1), (7, 6), (5, 100), (300, 512), (4, 1100)])
def test_join_widths(batch, d):
    """Single values, rows that share a CTA, a row per CTA, rows wider than a CTA."""
    seq, ns = torch.randn(batch, d, device="cuda"), torch.randn(batch, d, device="cuda")
    for cast_type, code in ((torch.bfloat16, _lib.BF16), (torch.float16, _lib.F16)):
        joined, cast = torch.empty(batch, 2 * d, device="cuda"), torch.empty(batch, 2 * d, dtype=cast_type, device="cuda")
        assert _lib.load().tb200_join_summaries(_p(seq), _p(ns), _p(joined), _p(cast), batch, d, code, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(joined, torch.cat([seq, ns], 1)) and torch.equal(cast, joined.to(cast_type))
