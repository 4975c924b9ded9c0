"""Codestreams written straight into Python bytes objects."""
import ctypes
import signal
import sys
import threading

import numpy as np
import pytest

import jp2lam_gb300 as jl
from jp2lam_gb300 import _native


def test_importing_leaves_pythonapi_prototypes_alone():
    for name in ("PyBytes_FromStringAndSize", "PyBytes_AsString"):
        f = getattr(ctypes.pythonapi, name)
        assert f.restype is ctypes.c_int and f.argtypes is None


def test_result_alloc_without_memory_returns_null():
    lib = _native.load_library()
    results = _native._Results(lib, 2)
    alloc = lambda i, n: lib.jp2g_py_result_alloc(ctypes.byref(results._results), i, n)  # noqa: E731
    for n in (1 << 62, 1 << 63, (1 << 64) - 1):
        assert alloc(0, n) is None
    assert alloc(2, 10) is None  # not an index of the call
    at = alloc(1, 5)
    ctypes.memmove(at, b"hello", 5)
    assert results.take(1) == b"hello"
    assert alloc(1, 0) and results.take(1) == b""


def test_result_objects_are_released_once():
    lib = _native.load_library()
    results = _native._Results(lib, 1)

    def new(n):  # an object in the slot, and this reference to it
        lib.jp2g_py_result_alloc(ctypes.byref(results._results), 0, n)
        return _native._new_ref(results._objects[0])

    first = new(1000)
    refs = sys.getrefcount(first)
    second = new(2000)  # replaces it
    assert sys.getrefcount(first) == refs - 1
    assert sys.getrefcount(second) == refs
    taken = results.take(0)
    assert taken is second and sys.getrefcount(second) == refs  # the slot's is now `taken`'s
    third = new(3000)
    with pytest.raises(KeyError), results:
        raise KeyError  # a call that fails leaves nothing behind
    assert sys.getrefcount(third) == refs - 1 and results._objects[0] is None
    fourth = new(4000)
    del results
    assert sys.getrefcount(second) == refs and sys.getrefcount(fourth) == refs - 1


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


def _raw_encode(eng, px, w, h, c, q):
    """jp2g_encode on an engine's context and jp2g_free, as a C caller has them."""
    out, n = _native._u8p(), ctypes.c_size_t()
    rc = eng.lib.jp2g_encode(eng.handle, px.ctypes.data_as(ctypes.c_void_p), w, h, c, 1, q, 0, ctypes.byref(out),
                             ctypes.byref(n))
    assert rc == 0
    data = ctypes.string_at(out, n.value)
    eng.lib.jp2g_free(out)
    return data


@pytest.mark.gpu
def test_raw_calls_on_an_engines_context_own_their_results(orc):
    w, h = 200, 150
    px = np.random.default_rng(2).integers(0, 256, w * h, dtype=np.uint8)
    want = orc.encode(px, w, h, 1, 80, 0)
    eng = jl.Engine(0)
    try:
        assert eng.encode(px, w, h, 1, 80, 0) == want
        assert _raw_encode(eng, px, w, h, 1, 80) == want
        raw = []

        def other():
            for _ in range(100):
                raw.append(_raw_encode(eng, px, w, h, 1, 80))

        t = threading.Thread(target=other)
        t.start()
        while t.is_alive():
            page = {"px": px, "w": w, "h": h, "ncomp": 1, "quality": 80, "fmt": 0}
            assert eng.encode_batch([page, page]) == [want, want]
        t.join()
        assert raw == [want] * 100
    finally:
        eng.close()


@pytest.mark.gpu
def test_result_alloc_of_a_context(orc):
    # a context's allocator: asked by the encode calls of any thread but the
    # engine's own and those with one of theirs; null ends it
    w, h = 120, 90
    px = np.random.default_rng(3).integers(0, 256, w * h, dtype=np.uint8)
    want = orc.encode(px, w, h, 1, 60, 0)
    eng = jl.Engine(0)
    memory = np.zeros(1 << 20, np.uint8)

    @_native._ResultAlloc
    def alloc(user, index, n):
        return memory.ctypes.data if index == 0 and n <= memory.size else None

    def raw():
        out, n = _native._u8p(), ctypes.c_size_t()
        rc = eng.lib.jp2g_encode(eng.handle, px.ctypes.data_as(ctypes.c_void_p), w, h, 1, 1, 60, 0,
                                 ctypes.byref(out), ctypes.byref(n))
        assert rc == 0
        return ctypes.cast(out, ctypes.c_void_p).value, n.value

    try:
        assert eng.lib.jp2g_set_result_alloc(eng.handle, alloc, None) == 0
        at, n = raw()
        assert at == memory.ctypes.data and memory[:n].tobytes() == want
        memory[:n] = 0
        assert eng.encode(px, w, h, 1, 60, 0) == want
        assert not memory[:n].any()
        assert eng.lib.jp2g_set_result_alloc(eng.handle, None, None) == 0
        assert _raw_encode(eng, px, w, h, 1, 60) == want
    finally:
        eng.close()
