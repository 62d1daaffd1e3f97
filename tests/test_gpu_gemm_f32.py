"""fp32 GEMM on the tensor cores (three-part bf16 operands) against float64 products.  Every product is right to about 2^-23 and the sums
accumulate in fp32: an fp32 GEMM errs by up to (K + 2) 2^-24 sum |a| |w|; twice that leaves room for the dropped products.  That worst
case is far above what an fp32 GEMM shows and would admit fewer parts; `test_no_further_from_float64_than_an_fp32_gemm` does not."""
from __future__ import annotations

import ctypes

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


@pytest.mark.parametrize("m", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("groups,n,k", [(1, 128, 64), (3, 384, 128), (1, 640, 1536)])
def test_against_float64(m, groups, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    a, w, b, r = rand(groups, m, k) * torch.exp(2 * rand(groups, m, k)), rand(groups, n, k), rand(groups, n), rand(groups, m, n)
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
    lib = _lib.load()
    split = torch.empty(groups, n, 3 * k, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.tb200_split_f32_weights(p(w), p(split), groups * n, k, None) == 0
    exact = torch.einsum("gmk,gnk->gmn", a.double(), w.double())
    bound = 2 * (k + 2) * 2.0 ** -24 * torch.einsum("gmk,gnk->gmn", a.abs().double(), w.abs().double())
    out = torch.empty(groups, m, n, device="cuda")
    assert lib.tb200_gemm_f32_grouped(p(a), p(split), None, None, p(out), groups, m, n, k, 0, p(status), None) == 0
    torch.cuda.synchronize()
    assert int(status) == 0 and bool(((out.double() - exact).abs() <= bound).all())
    assert lib.tb200_gemm_f32_grouped(p(a), p(split), p(b), p(r), p(r), groups, m, n, k, 1, p(status), None) == 0      # in place on the residual
    torch.cuda.synchronize()
    pre = out.double() + b[:, None].double()
    g2 = torch.Generator(device="cuda").manual_seed(m + n)
    res = [torch.randn(*s, device="cuda", generator=g2) for s in ((groups, m, k), (groups, m, k), (groups, n, k), (groups, n), (groups, m, n))][-1].double()
    want = pre * torch.sigmoid(pre) + res
    assert bool(((r.double() - want).abs() <= 1e-6 + 4e-6 * (pre.abs() + res.abs())).all())


def _product(a, w):
    m, k, n = a.shape[0], a.shape[1], w.shape[0]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    lib = _lib.load()
    split, out = torch.empty(n, 3 * k, dtype=torch.bfloat16, device="cuda"), torch.empty(m, n, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.tb200_split_f32_weights(p(w), p(split), n, k, None) == 0
    assert lib.tb200_gemm_f32_grouped(p(a), p(split), None, None, p(out), 1, m, n, k, 0, p(status), None) == 0
    torch.cuda.synchronize()
    assert int(status) == 0
    return out


@pytest.mark.parametrize("k", [64, 128, 256, 512, 2560])
@pytest.mark.parametrize("kind", ["normal", "wide", "positive"])
def test_no_further_from_float64_than_an_fp32_gemm(k, kind):
    """The form that this GEMM replaced is the library's SGEMM: its distance from the float64 product, on the same operands, is the
    bound (2-norm and largest element; both errors are sums of some 4e5 independent roundings, so a tenth covers their spread)."""
    g = torch.Generator(device="cuda").manual_seed(k)
    a, w = torch.randn(1000, k, device="cuda", generator=g), torch.randn(384, k, device="cuda", generator=g)
    if kind == "wide":
        a = a * torch.exp(2 * torch.randn(1000, k, device="cuda", generator=g))
    if kind == "positive":       # no cancellation: an accumulator that cuts off instead of rounding shows as a bias
        a, w = a.abs(), w.abs()
    exact = a.double() @ w.double().t()
    old = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        theirs = (a @ w.t()).double() - exact
    finally:
        torch.backends.cuda.matmul.allow_tf32 = old
    ours = _product(a, w).double() - exact
    assert ours.norm() <= 1.1 * theirs.norm()
    assert ours.abs().max() <= 2 * theirs.abs().max()


@pytest.mark.parametrize("m,k", [(1, 64), (129, 64), (1000, 128), (40_000, 64)])
def test_rows_without_a_split(m, k):
    """A value that is not finite, or rounds to an infinite bf16, gives the row what fp32 arithmetic gives; the rows beside it keep
    their results.  The longest case has several tiles per CTA, so that the marks of one tile are reused."""
    g = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, k, device="cuda", generator=g), torch.randn(256, k, device="cuda", generator=g)
    rows = torch.arange(0, m, 97, device="cuda")
    values = torch.tensor([float("inf"), float("-inf"), 3.4e38, float("nan")], device="cuda")[torch.arange(rows.numel(), device="cuda") % 4]
    a[rows, rows % k] = values
    w[:, :] = torch.where(w.abs() < 0.1, 0.1, w)      # no product of an infinity with nearly nothing
    clean = _product(torch.where(a.abs() < 1e30, a, 0.0), w)
    got = _product(a, w)
    keep = torch.ones(m, dtype=torch.bool, device="cuda")
    keep[rows] = False
    assert torch.equal(got[keep], clean[keep])
    want = a[rows].double() @ w.double().t()
    want = torch.where(want.abs() > 3.4028235e38, torch.sign(want) * float("inf"), want)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got[rows]), torch.isnan(want))
    assert torch.equal(got[rows][torch.isinf(want)].double(), want[torch.isinf(want)])
    torch.testing.assert_close(got[rows][finite].double(), want[finite], rtol=1e-5, atol=0)
