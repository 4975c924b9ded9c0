"""The MQ coder where its byte output is hard: contents whose code-blocks
end at every symbol count, carry through bytes of 0xFF, shift by many bits at
once or hardly at all, in every packing of blocks to a warp's lanes, against
the oracle."""
import ctypes

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


def _stop_content(kind, w, h, c):
    rng = np.random.default_rng(w + 7 * h + 31 * c)
    y, x = np.mgrid[0:h, 0:w]
    if kind == "faint":  # slopes too small to settle lambda: every pass is coded
        px = 128 + rng.integers(0, 2, (h, w, c))
    elif kind == "outlier":  # one huge coefficient above much small detail
        px = 120 + rng.integers(-6, 7, (h, w, c))
        px[h // 2, w // 2] = 255
        px[h // 3:h // 3 + 2, w // 5] = 0
    elif kind == "texture":
        px = 128 + 60 * np.sin(x / 3.1)[..., None] * np.cos(y / 4.7)[..., None] + rng.normal(0, 12, (h, w, c))
    else:  # chroma much fainter than luma
        g = np.where((x // 9 + y // 7) % 2, 230, 20)[..., None]
        px = g + rng.integers(0, 3, (h, w, c))
    return np.ascontiguousarray(np.clip(px, 0, 255).astype(np.uint8))


@pytest.mark.parametrize("kind", ["faint", "outlier", "texture", "checks"])
@pytest.mark.parametrize("w,h,c", [(64, 64, 1), (200, 150, 3), (321, 257, 1)])
def test_blocks_stopped_early_lose_nothing(eng, orc, kind, w, h, c):
    # lossy codestreams of blocks whose coding stops at some bit-plane, over
    # the whole range of lambda, byte for byte
    px = _stop_content(kind, w, h, c)
    for q in (0, 1, 5, 15, 29, 30, 45, 50, 70, 85, 92, 98, 99):
        assert eng.encode(px, w, h, c, q, 0) == orc.encode(px, w, h, c, q, 0), q


def test_block_inspection_shows_every_pass(eng, orc):
    # jp2g_debug_blocks reports complete coding, an encode only what it needed
    w, h = 256, 256
    px = _stop_content("texture", w, h, 1)
    rows = eng.debug_blocks(px, w, h, 1, 60)
    coded = rows[:, 0] > 0
    assert np.array_equal(rows[coded, 2], 1 + 3 * (rows[coded, 0] - 1))
    full = eng.counters()[2]
    eng.encode(px, w, h, 1, 60, 0)
    assert 0 < eng.counters()[2] < full


def test_second_round_of_a_large_wave(eng, orc):
    # a wave large enough that only the bit-planes foreseen are modelled at
    # first, of contents that mislead the forecast: sparse outliers over much
    # faint detail, chroma whose slopes never settle lambda, blocks of every
    # size; each page against the oracle
    pages, want = [], []
    kinds = ["outlier", "faint", "texture", "checks"]
    for i in range(28):
        w, h, c = (1024, 768, 3) if i % 7 == 0 else (640 + 7 * i, 512 + 5 * i, 1 + 2 * (i % 2))
        px = _stop_content(kinds[i % 4], w, h, c)
        q = (85, 50, 97, 30, 100)[i % 5]
        pages.append({"px": px, "w": w, "h": h, "ncomp": c, "quality": q, "fmt": 0})
    pages = pages * 4
    outs = eng.encode_batch(pages)
    assert eng.counters()[0] > 48 * 152
    for i in range(28):
        p = pages[i]
        ref = orc.encode(p["px"], p["w"], p["h"], p["ncomp"], p["quality"], 0)
        for r in range(4):
            assert outs[i + 28 * r] == ref, (i, r)


@pytest.mark.parametrize("q", [100, 75])
@pytest.mark.parametrize("kind", ["flat", "noise", "one", "halves"])
def test_split_wave(eng, orc, kind, q):
    # a wave just large enough to be coded in two parts: nothing to code, every
    # block in the first part, all but one in the second, and both alike
    w, h = 2303, 2245
    img = np.full((h, w), 128, np.uint8)
    rng = np.random.default_rng(5)
    if kind == "noise":
        img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    elif kind == "one":
        img[700:760, 900:960] = rng.integers(0, 256, (60, 60))
    elif kind == "halves":
        img[:, : w // 2] = rng.integers(0, 256, (h, w // 2))
        img[:, w // 2:] = rng.integers(126, 130, (h, w - w // 2))
    data = eng.encode(img.ravel(), w, h, 1, q, 0)
    assert eng.counters()[0] > 8 * 152
    assert data == orc.encode(img.ravel(), w, h, 1, q, 0)


@pytest.mark.parametrize("q", [20, 50, 95, 99])
@pytest.mark.parametrize("kind", ["noise", "sparse", "ramp"])
@pytest.mark.parametrize("w,h,c", [(64, 64, 1), (2200, 1800, 3)])
def test_hulls_by_warps_and_by_lanes(eng, orc, kind, w, h, c, q):
    # rate-distortion curves of few and of many passes, in a wave of one block
    # and in one whose blocks are too many for a warp each
    px = np.repeat(_content(kind, w, h).reshape(h, w, 1), c, axis=2).ravel()
    data = eng.encode(px, w, h, c, q, 0)
    assert (eng.counters()[0] > 16 * 152) == (w > 64)
    assert data == orc.encode(px, w, h, c, q, 0)


def _round_counters(eng):
    """Bit-planes modelled, blocks left unfinished by the first round, blocks
    coded on in the second."""
    c = (ctypes.c_uint64 * 11)()
    assert eng.lib.jp2g_counters(eng.handle, c, 11) == 11
    return list(c[8:])


def _misleading(w, h, seed):
    """Content whose bit counts make coding look dearer than it is: every block
    regular (signs and bits that the contexts foresee), so that many more
    bit-planes are worth their bytes than a forecast from counts expects."""
    y, x = np.mgrid[0:h, 0:w]
    period = 2 + seed % 3
    px = 128 + (((x // period + y // period) & 1) * 2 - 1) * (20 + 7 * (seed % 5)) + ((x ^ y) & 3)
    return px.astype(np.uint8)


@pytest.mark.parametrize("q", [20, 60, 90])
def test_second_round_is_taken(eng, orc, q):
    # 32x32 and 64x64 blocks; some blocks of the wave are left unfinished by the
    # first round, and some of these are coded on by the second
    pages = []
    for i in range(40):
        w, h = (1024 + 3 * i, 900 + i) if q < 30 else (2048 + 3 * i, 1500 + i)
        px = _misleading(w, h, i) if i % 2 else _stop_content(("outlier", "texture")[i // 2 % 2], w, h, 1)
        pages.append({"px": px, "w": w, "h": h, "ncomp": 1, "quality": q, "fmt": 0})
    outs = eng.encode_batch(pages)
    assert eng.counters()[0] > 48 * 152
    modelled, unfinished, again = _round_counters(eng)
    assert modelled > 0
    assert unfinished >= again > 0
    for i in range(0, 40, 3):
        p = pages[i]
        assert outs[i] == orc.encode(p["px"], p["w"], p["h"], 1, q, 0, threads=8), i


@pytest.mark.parametrize("bpw", [1, 3, 31, 32])
@pytest.mark.parametrize("large", [False, True])
def test_packings_of_split_and_large_waves(eng, orc, bpw, large):
    # a packing of the caller's choice where the wave is coded in two parts, and
    # where there is a second round
    rng = np.random.default_rng(bpw)
    pages = []
    for i in range(12 if large else 4):
        w, h = (1800 + 5 * i, 1500 + i) if large else (1600, 1300 + i)
        px = _misleading(w, h, i)
        px[: h // 3] = rng.integers(0, 256, (h // 3, w))
        pages.append({"px": px, "w": w, "h": h, "ncomp": 1, "quality": 70, "fmt": 0})
    if large:
        pages = pages + pages[:1] * 2
    eng.set_option(_native.OPT_MQ_BLOCKS_PER_WARP, bpw)
    try:
        outs = eng.encode_batch(pages)
    finally:
        eng.set_option(_native.OPT_MQ_BLOCKS_PER_WARP, 0)
    blocks = eng.counters()[0]
    assert blocks > 48 * 152 if large else 8 * 152 < blocks <= 48 * 152
    assert (_round_counters(eng)[2] > 0) == large
    for p, out in list(zip(pages, outs))[::3]:
        assert out == orc.encode(p["px"], p["w"], p["h"], 1, 70, 0, threads=8)


def test_second_round_of_most_blocks(eng, orc):
    # more blocks in the second round than its warps have lanes: each CTA codes several lists
    w, h = 1700, 2200
    y, x = np.mgrid[0:h, 0:w]
    px = ((((x // 2 + y // 2) & 1) * 60 + 100) + ((x ^ y) & 3)).astype(np.uint8)
    outs = eng.encode_batch([{"px": px, "w": w, "h": h, "ncomp": 1, "quality": 20, "fmt": 0}] * 32)
    assert _round_counters(eng)[2] > 152 * 4 * 4 * 32
    assert set(outs) == {orc.encode(px, w, h, 1, 20, 0, threads=8)}
