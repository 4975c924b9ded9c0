"""Codestreams written straight into Python bytes objects."""
import ctypes
import signal
import sys

import numpy as np
import pytest

import jp2lam_gb300 as jl
from jp2lam_gb300 import _native


def test_importing_leaves_pythonapi_prototypes_alone():
    for name in ("PyBytes_FromStringAndSize", "PyBytes_AsString"):
        f = getattr(ctypes.pythonapi, name)
        assert f.restype is ctypes.c_int and f.argtypes is None


class _NoEngine:
    """As much of an Engine as _Results needs without a GPU."""
    handle = None

    def __init__(self):
        self.lib = _native.load_library()


def test_result_alloc_without_memory_returns_null():
    eng = _NoEngine()
    results = _native._Results(eng, 2)
    alloc = lambda i, n: eng.lib.jp2g_py_result_alloc(ctypes.byref(results._results), i, n)  # noqa: E731
    for n in (1 << 62, 1 << 63, (1 << 64) - 1):
        assert alloc(0, n) is None
    assert alloc(2, 10) is None  # not an index of the call
    at = alloc(1, 5)
    ctypes.memmove(at, b"hello", 5)
    assert results[1] == b"hello"
    assert alloc(1, 0) and results[1] == b""


def test_result_objects_are_released_once():
    eng = _NoEngine()
    results = _native._Results(eng, 1)
    alloc = lambda n: eng.lib.jp2g_py_result_alloc(ctypes.byref(results._results), 0, n)  # noqa: E731
    alloc(1000)
    first = results[0]
    mine = sys.getrefcount(first) - 1  # without the slot's
    alloc(2000)
    assert sys.getrefcount(first) == mine
    second = results[0]
    with_slot = sys.getrefcount(second)
    del results
    assert sys.getrefcount(second) == with_slot - 1


@pytest.mark.gpu
def test_signal_handler_that_raises_during_an_encode():
    # the handler's exception leaves the call; before and after it, codestreams
    class Interrupt(Exception):
        pass

    def handler(*_):
        raise Interrupt

    w, h = 5100, 6600
    px = np.random.default_rng(1).integers(0, 256, w * h, dtype=np.uint8)
    eng = jl.Engine(0)
    before = signal.signal(signal.SIGALRM, handler)
    try:
        want = eng.encode(px, w, h, 1, 100, 0)
        for delay in (0.0005, 0.002, 0.004):
            with pytest.raises(Interrupt):
                signal.setitimer(signal.ITIMER_REAL, delay)
                while True:
                    eng.encode(px, w, h, 1, 100, 0)
            assert eng.encode(px, w, h, 1, 100, 0) == want
    finally:
        signal.setitimer(signal.ITIMER_REAL, 0)
        signal.signal(signal.SIGALRM, before)
        eng.close()
