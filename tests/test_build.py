"""The host library beside the CUDA library."""
import sysconfig

import numpy as np
import pytest

from apt_serve_b200 import _native as N
from apt_serve_b200 import build as B
from apt_serve_b200.device_metadata import pack_tables


def test_the_host_library_is_named_after_the_interpreter():
    """It inlines the layout of lists and integers: built for one interpreter, it reads wrong values under another."""
    assert N.HOST_LIB_PATH == B.HOST_LIB_PATH
    assert N.HOST_LIB_PATH.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert sysconfig.get_config_var("SOABI") in N.HOST_LIB_PATH.name


@pytest.mark.parametrize("compiler", ["false", "/nonexistent/compiler"])
def test_no_host_compiler_is_no_obstacle(monkeypatch, tmp_path, capsys, compiler):
    """Without g++ or Python.h the CUDA library is built all the same and the tables are packed by numpy, with the same result."""
    monkeypatch.setenv("CXX", compiler)
    monkeypatch.setattr(B, "HOST_LIB_PATH", tmp_path / "host.so")
    monkeypatch.setattr(B, "LIB_DIR", tmp_path)
    monkeypatch.setattr(B, "build_cuda", lambda force, verbose: B.LIB_PATH)
    assert B.build(force=True) == B.LIB_PATH
    assert not B.HOST_LIB_PATH.exists() and "not built" in capsys.readouterr().err

    tables, shared, hid = [[5, 6, 7], (1,), [], [2 ** 31 - 1]], [[9], [], [4, 4], [8, 0, 3]], np.array([True, False, True, True])
    packed = []
    for path in (N.HOST_LIB_PATH, B.HOST_LIB_PATH):
        monkeypatch.setattr(N, "HOST_LIB_PATH", path)
        monkeypatch.setattr(N, "_host_lib", None)
        out = np.full((3, 4, 3), -9, dtype=np.int32)
        pack_tables(tables, shared, hid, *out)
        packed.append(out)
    assert N.host_lib() is None
    assert np.array_equal(*packed) and packed[0][2].tolist() == [[9, 0, 0], [1, 0, 0], [4, 4, 0], [8, 0, 3]]
