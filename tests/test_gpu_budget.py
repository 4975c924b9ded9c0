"""Calls under a device memory budget whose pools are full of earlier calls'."""
import numpy as np
import pytest

import jp2lam_gb300 as jl

pytestmark = pytest.mark.gpu

W, H = 1000, 700


def _page(seed):
    return np.random.default_rng(seed).integers(0, 256, W * H, dtype=np.uint8)


@pytest.fixture()
def full():
    # 40 MB hold a page's encode (36 MB of pools) or a file's decode (7 MB)
    e = jl.Engine(0, 40_000_000)
    e.encode(_page(1), W, H, 1, 75, 0)
    yield e
    e.close()


def test_decode_after_an_encode_that_filled_the_budget(full, orc):
    data = orc.encode(_page(2), W, H, 1, 75, 0)
    want = orc.decode(data)[3]
    assert np.array_equal(np.asarray(full.decode(data)[0]), want)
    full.encode(_page(1), W, H, 1, 75, 0)
    assert all(np.array_equal(np.asarray(g[0]), want) for g in full.decode_batch([data] * 3))
    assert full.encode(_page(2), W, H, 1, 75, 0) == data


def test_metrics_after_an_encode_that_filled_the_budget(full, orc):
    w, h = 700, 600
    px = _page(3)[: w * h]
    data, psnr, ssim = full.encode_with_psnr(px, w, h, 1, 75, 0)
    assert data == orc.encode(px, w, h, 1, 75, 0)
    want = orc.quality_metrics(px, w, h, 1, 75)
    assert abs(psnr - want[0]) < 1e-6 and abs(ssim - want[1]) < 1e-9
