"""The MQ coder where its byte output is hard: contents whose code-blocks
end at every symbol count, carry through bytes of 0xFF, shift by many bits at
once or hardly at all, in every packing of blocks to a warp's lanes, against
the oracle."""
import numpy as np
import pytest

import jp2lam_gb300 as jl
from jp2lam_gb300 import _native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = jl.Engine(0)
    yield e
    e.close()


def _content(kind, w, h):
    rng = np.random.default_rng(w * 1009 + h)
    if kind == "noise":
        return rng.integers(0, 256, (h, w), dtype=np.uint8)
    if kind == "binary":
        return np.where(rng.random((h, w)) < 0.5, 0, 255).astype(np.uint8)
    if kind == "sparse":  # long runs of the most probable symbol, then surprises
        return np.where(rng.random((h, w)) < 0.002, 255, 128).astype(np.uint8)
    if kind == "flat":
        return np.full((h, w), 255, np.uint8)
    x = np.arange(w)[None, :] * 3 + np.arange(h)[:, None] * 5
    return (x & 0xff).astype(np.uint8)


@pytest.mark.parametrize("kind", ["noise", "binary", "sparse", "flat", "ramp"])
@pytest.mark.parametrize("w,h", [(1, 1), (4, 4), (63, 65), (64, 64), (129, 100), (257, 300)])
def test_bytes_equal_the_oracle(eng, orc, kind, w, h):
    px = _content(kind, w, h)
    for q in (100, 97, 60, 10):
        assert eng.encode(px, w, h, 1, q, 0) == orc.encode(px, w, h, 1, q, 0)


@pytest.mark.parametrize("bpw", [0, 1, 3, 31, 32])
def test_lanes_of_a_warp_do_not_disturb_each_other(eng, orc, bpw):
    # blocks of very different weight side by side: some lanes end long before others
    w, h = 420, 390
    px = _content("sparse", w, h)
    px[100:230, 60:250] = _content("noise", 190, 130)
    eng.set_option(_native.OPT_MQ_BLOCKS_PER_WARP, bpw)
    try:
        for q in (100, 90, 25):
            assert eng.encode(px, w, h, 1, q, 1) == orc.encode(px, w, h, 1, q, 1)
    finally:
        eng.set_option(_native.OPT_MQ_BLOCKS_PER_WARP, 0)
