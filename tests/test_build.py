"""The host library beside the CUDA library."""
import sysconfig

from apt_serve_b200 import _native as N
from apt_serve_b200 import build as B


def test_the_host_library_is_named_after_the_interpreter():
    """It inlines the layout of lists and integers: built for one interpreter, it reads wrong values under another."""
    assert N.HOST_LIB_PATH == B.HOST_LIB_PATH
    assert N.HOST_LIB_PATH.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert sysconfig.get_config_var("SOABI") in N.HOST_LIB_PATH.name
