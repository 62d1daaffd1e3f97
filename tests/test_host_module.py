"""The host module (``_native.so``): how it is built, and the operators without it."""
from __future__ import annotations

import time
from pathlib import Path

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200 import _lib, build, ops


def test_it_shares_the_cxx_runtime_of_torch():
    """With a runtime of its own, an error message that prints one of torch's types ended the process."""
    if not build.NATIVE_PATH.exists():
        pytest.skip("the host module is not built")
    data = build.NATIVE_PATH.read_bytes()
    assert b"\0libstdc++.so.6\0" in data                       # among the needed libraries
    assert b"_txnal_logic_error_get_msg" not in data           # defined by libstdc++ itself


def _unloadable():
    raise RuntimeError("the host module does not load")


@pytest.mark.parametrize("library,module", [(False, True), (True, False), (False, False)])
def test_arguments_are_looked_at_first(monkeypatch, library, module):
    """With the library, the host module or both missing, a wrong argument is still a ValueError, and the rest a RuntimeError."""
    monkeypatch.setattr(ops, "_host", ops._LazyHost())
    monkeypatch.setattr(_lib, "library_available", lambda: library)
    if not module:
        monkeypatch.setattr(_lib, "native", _unloadable)
    for _ in range(2):
        with pytest.raises(ValueError, match="at least 2 dimensions"):
            ops.rms_norm(torch.ones(4), torch.ones(4))
        with pytest.raises(ValueError, match="matching head counts"):
            ops.flash_attention(torch.ones(1, 2, 4, 64), torch.ones(1, 3, 4, 64), torch.ones(1, 3, 4, 64))
        with pytest.raises(RuntimeError):
            ops.rms_norm(torch.ones(2, 4), torch.ones(4))


@pytest.mark.gpu
def test_operators_run_without_the_host_module(monkeypatch):
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = torch.randn(33, 64, device="cuda", generator=g), torch.rand(64, device="cuda", generator=g)
    ids = torch.randint(0, 50, (9, 4), device="cuda", generator=g)
    q, k, v = (torch.randn(2, 2, 40, 64, device="cuda", generator=g).bfloat16() for _ in range(3))

    def results():
        xr = x.clone().requires_grad_()
        y = ops.rms_norm(xr, w)
        y.sum().backward()
        return (y.detach(), xr.grad, ops.layer_norm(x, w, w, pre_silu=True), ops.embedding_bag_mean(torch.outer(w.repeat(2), w)[:50].contiguous(), ids),
                ops.flash_attention(q, k, v, is_causal=True), ops.varlen_attention(q, k, v, ns_start=40))

    want = results()
    monkeypatch.setattr(ops, "_host", ops._LazyHost())
    monkeypatch.setattr(_lib, "native", _unloadable)
    for a, b in zip(results(), want):
        assert torch.equal(a, b)


def test_another_torch_makes_the_host_objects_stale(monkeypatch, tmp_path):
    commands = []
    monkeypatch.setattr(build, "BUILD", tmp_path)

    def run(cmd, what, verbose):
        commands.append(what)
        Path(cmd[-1]).write_bytes(b"")

    monkeypatch.setattr(build, "_run", run)
    src = next(iter(sorted(build.HOST.glob("*.cpp"))))

    def compiled() -> int:
        commands.clear()
        build._compile_host(src, build._host_toolchain(), False)
        return len(commands)

    assert compiled() == 1
    assert compiled() == 0
    time.sleep(0.02)       # file times
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert compiled() == 1
    assert compiled() == 0
    time.sleep(0.02)
    monkeypatch.undo()     # back to the first one: its objects are gone
    monkeypatch.setattr(build, "BUILD", tmp_path)
    monkeypatch.setattr(build, "_run", run)
    assert compiled() == 1
