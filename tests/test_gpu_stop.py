"""Blocks whose coding stops early, where the largest slope of a component is
near one that settles lambda (or a share of it): codestreams byte for byte
against the oracle."""
import numpy as np
import pytest

import jp2lam_gb300 as jl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = jl.Engine(0)
    yield e
    e.close()


def _regular_page(orc, seed):
    """A gray page of one level: an LL block of a single bit-plane, all ones, and
    an HH block of two or three with much smaller slopes."""
    rng = np.random.default_rng(seed)
    w, h, q = (int(v) for v in (rng.integers(50, 64), rng.integers(54, 64), rng.integers(12, 19)))
    _, step, _ = orc.coefficients_f64(np.full(w * h, 128, np.uint8), w, h, 1, q, 0)
    lw, lh = (w + 1) // 2, (h + 1) // 2
    co = np.zeros((h, w), np.float32)
    co[:lh, :lw] = 1.5
    density, larger, minus = rng.uniform(.65, 1), rng.uniform(0, .3), rng.uniform(0, .4)
    n = (h - lh, w - lw)
    v = rng.integers(2, 4) + (rng.random(n) < larger) + .5
    co[lh:, lw:] = (rng.random(n) < density) * np.where(rng.random(n) < minus, -1, 1) * v
    px = orc.dwt((co * step).ravel(), w, h, 1, 97, inverse=True) + 128
    return np.clip(np.rint(px), 0, 255).astype(np.uint8), w, h, q


# a share of lambda that only the LL block's last pass, before its termination,
# would have shown
@pytest.mark.parametrize("seed", [37, 55, 139, 248, 1097, 2432, 11635, 64440, 139056, 155534])
def test_last_pass_shows_no_slope(eng, orc, seed):
    px, w, h, q = _regular_page(orc, seed)
    assert eng.encode(px, w, h, 1, q, 0) == orc.encode(px, w, h, 1, q, 0)
