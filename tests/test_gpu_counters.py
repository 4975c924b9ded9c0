"""Work counters of an encode against what ran on the device."""
import numpy as np
import pytest

import jp2lam_gb300 as jl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = jl.Engine(0)
    yield e
    e.close()


def _kernels(call):
    """Kernels launched on the device during a call."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.init()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return [n for n in names if not n.startswith(("Memcpy", "Memset"))]


@pytest.fixture(scope="module", autouse=True)
def profiler():
    import torch

    fill = lambda: torch.zeros(64, device="cuda").add_(1)  # noqa: E731
    _kernels(fill)  # a process's first profile misses what it runs
    if not _kernels(fill):
        pytest.skip("no profile of kernels here")


# waves of few blocks; of more than a scan's 1024; of one thread row (levels
# run alone); split in two parts
@pytest.mark.parametrize("w,h,c,q", [(64, 64, 1, 80), (256, 256, 1, 100), (700, 1, 1, 70), (1600, 1500, 3, 90),
                                     (3000, 3300, 1, 85)])
def test_kernel_launches_of_a_page(eng, w, h, c, q):
    px = np.random.default_rng(w).integers(0, 256, w * h * c, dtype=np.uint8)
    eng.encode(px, w, h, c, q, 0)
    names = _kernels(lambda: eng.encode(px, w, h, c, q, 0))
    assert len(names) == eng.counters()[5], names


def test_kernel_launches_of_a_large_wave(eng):
    # more than 1024 pages and packets, and a second round
    rng = np.random.default_rng(9)
    pages = [{"px": rng.integers(0, 256, 160 * 130, dtype=np.uint8), "w": 160, "h": 130, "ncomp": 1, "quality": 80,
              "fmt": 0} for _ in range(1100)]
    eng.encode_batch(pages)
    names = _kernels(lambda: eng.encode_batch(pages))
    assert eng.counters()[0] > 48 * 152
    assert len(names) == eng.counters()[5], names


@pytest.mark.parametrize("w,h,split", [(1000, 900, False), (3000, 3300, True)])
def test_stage_times_of_modelling_and_coding(eng, w, h, split):
    # a split wave's first part (here the noise) is coded while the second is
    # modelled (the much fainter rest of the page)
    rng = np.random.default_rng(w)
    px = rng.integers(100, 156, (h, w), dtype=np.uint8)
    px[:, : w // 4] = rng.integers(0, 256, (h, w // 4))
    eng.set_timing(True)
    try:
        eng.encode(px, w, h, 1, 85, 0)
        eng.encode(px, w, h, 1, 85, 0)
        t = eng.stage_times()
    finally:
        eng.set_timing(False)
    assert (eng.counters()[0] > 8 * 152) == split
    beside = t["t1_analyze"] + t["t1_model"] + t["t1_mq"] - t["tier1"]
    assert beside > 0.02 * t["tier1"] if split else abs(beside) < 0.01 * t["tier1"]
    assert t["t1_mq"] < t["tier1"]
