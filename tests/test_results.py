"""Codestreams written straight into Python bytes objects."""
import ctypes

import jp2lam_gb300  # noqa: F401


def test_importing_leaves_pythonapi_prototypes_alone():
    for name in ("PyBytes_FromStringAndSize", "PyBytes_AsString"):
        f = getattr(ctypes.pythonapi, name)
        assert f.restype is ctypes.c_int and f.argtypes is None
