"""The host module (``_native.so``) as it was built."""
from __future__ import annotations

import pytest

from taac_2026_b200 import build


def test_it_shares_the_cxx_runtime_of_torch():
    """With a runtime of its own, an error message that prints one of torch's types ended the process."""
    if not build.NATIVE_PATH.exists():
        pytest.skip("the host module is not built")
    data = build.NATIVE_PATH.read_bytes()
    assert b"\0libstdc++.so.6\0" in data                       # among the needed libraries
    assert b"_txnal_logic_error_get_msg" not in data           # defined by libstdc++ itself
