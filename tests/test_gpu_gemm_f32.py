"""fp32 GEMM on the tensor cores (three-part bf16 operands) against float64 products.  Every product is right to about 2^-23 and the sums
accumulate in fp32: an fp32 GEMM errs by up to (K + 2) 2^-24 sum |a| |w|; twice that leaves room for the dropped products."""
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
