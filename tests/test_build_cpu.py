"""The built extension as a file."""
import os

import pytest

from slapo_b200.ops import native


@pytest.mark.skipif(not os.path.exists(native.lib_path()), reason="extension not built")
def test_one_cpp_runtime_in_the_process():
    """The extension uses the process's libstdc++: with a copy of its own, formatting a number
    into an error message crashes."""
    with open(native.lib_path(), "rb") as f:
        assert b"libstdc++.so.6\0" in f.read()
