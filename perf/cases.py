"""The engine's work as its users have it done, for timing and comparison.

Every case is one call of the public API: single pages, batches and decoding,
from a 256x256 thumbnail to a 5100x6600 scan, gray and sRGB, lossy and
lossless. Pages are document-like: text lines of the repository's seeded
page generator and, on most, a photo (blurred noise, as the generator's).

listed() and draw(rng) give cases, prepare(case, seed) what a program holds
before the call, run(state) makes the call, work(case) states the bytes and
operations it cannot do without.
"""
import concurrent.futures
import math
import os

import numpy as np
import torch

import jp2lam_gb300 as jl
from jp2lam_gb300._native import default_engine, synth_page

# Page sizes of the mixed batches: half, full and double letter pages at
# 150 to 600 dpi, the thumbnail of the served mix, and a ragged crop.
MIX = [(256, 256), (517, 389), (1275, 1650), (2550, 3300), (3400, 4400)]
MIX_QUALITY = [50, 75, 85, 100]


def listed():
    return [
        # a thumbnail on its own: the smallest call, latency and launches
        {"name": "encode_thumb", "do": "encode", "w": 256, "h": 256, "ncomp": 1, "quality": 60, "fmt": 1, "n": 1,
         "photo": 0.3},
        # a crop of ragged size, small and in colour, as a bare codestream
        {"name": "encode_odd_rgb", "do": "encode", "w": 517, "h": 389, "ncomp": 3, "quality": 85, "fmt": 0, "n": 1,
         "photo": 0.3},
        # one scanned gray page at the default quality: the headline call
        {"name": "encode_page_gray", "do": "encode", "w": 2550, "h": 3300, "ncomp": 1, "quality": 85, "fmt": 1,
         "n": 1, "photo": 0.057},
        # the same page in colour at a web quality
        {"name": "encode_page_rgb", "do": "encode", "w": 2550, "h": 3300, "ncomp": 3, "quality": 75, "fmt": 1,
         "n": 1, "photo": 0.057},
        # an archive scan at 600 dpi, lossless: the largest single page
        {"name": "encode_scan_lossless", "do": "encode", "w": 5100, "h": 6600, "ncomp": 3, "quality": 100, "fmt": 1,
         "n": 1, "photo": 0.1},
        # encoding with the quality metrics computed beside it
        {"name": "encode_psnr_rgb", "do": "psnr", "w": 1275, "h": 1650, "ncomp": 3, "quality": 62, "fmt": 1, "n": 1,
         "photo": 0.1},
        # many thumbnails in one call
        {"name": "batch_thumbs", "do": "batch", "w": 256, "h": 256, "ncomp": 1, "quality": 60, "fmt": 1, "n": 48,
         "photo": 0.3},
        # a document of equal colour pages already on the GPU
        {"name": "batch_pages_rgb", "do": "batch_device", "w": 2550, "h": 3300, "ncomp": 3, "quality": 75, "fmt": 1,
         "n": 24, "photo": 0.057},
        # pages of mixed size, colour and quality from host memory
        {"name": "batch_mixed", "do": "batch_mixed", "n": 24, "photo": 0.1},
        # opening a small lossless file
        {"name": "decode_tile_lossless", "do": "decode", "w": 512, "h": 512, "ncomp": 1, "quality": 100, "fmt": 0,
         "n": 1, "photo": 0.3},
        # opening one gray page
        {"name": "decode_page_gray", "do": "decode", "w": 2550, "h": 3300, "ncomp": 1, "quality": 85, "fmt": 1,
         "n": 1, "photo": 0.057},
        # reading a document back: equal colour pages in one call
        {"name": "decode_batch_rgb", "do": "decode", "w": 2550, "h": 3300, "ncomp": 3, "quality": 75, "fmt": 1,
         "n": 12, "photo": 0.057},
    ]


def draw(rng):
    do = rng.choice(["encode", "encode", "encode", "psnr", "batch", "batch_device", "batch_mixed", "decode", "decode",
                     "decode"])
    photo = round(rng.uniform(0.0, 0.3), 3)
    if do == "batch_mixed":
        return {"do": do, "n": rng.randint(2, 20), "photo": photo}
    w = int(math.exp(rng.uniform(math.log(64), math.log(5100))))
    h = max(48, min(6600, int(w * math.exp(rng.uniform(math.log(0.6), math.log(1.6))))))
    ncomp = rng.choice([1, 3])
    # thumbnail and document presets, page and archive qualities
    quality = rng.choice([20, 30, 42, 50, 60, 62, 75, 85, 90, 95, 100])
    if do == "psnr":
        quality = min(quality, 95)  # lossless pages have no metrics to compute
    n = 1
    if do.startswith("batch") or (do == "decode" and rng.random() < 0.4):
        most = max(1, min(48, int(100e6 / (w * h * ncomp))))
        n = max(1, int(math.exp(rng.uniform(0.0, math.log(most + 0.5)))))
    return {"do": do, "w": w, "h": h, "ncomp": ncomp, "quality": quality, "fmt": rng.choice([0, 1]), "n": n,
            "photo": photo}


def _pages(case, seed):
    """Size, colour, quality and seed of each page of a case."""
    if case["do"] != "batch_mixed":
        return [(case["w"], case["h"], case["ncomp"], case["quality"], seed * 1000003 + 64 * i)
                for i in range(case["n"])]
    out = []
    for i in range(case["n"]):  # every size, both colours and all qualities in turn
        w, h = MIX[i % len(MIX)]
        out.append((w, h, 1 if (i // 2) % 2 == 0 else 3, MIX_QUALITY[(i + i // 4) % 4], seed * 1000003 + 64 * i))
    return out


def _photo(w, h, ncomp, seed):
    """White noise blurred with a sigma = 8 kernel, rescaled to +/-60 around 128."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed & 0x7FFFFFFF)
    x = torch.rand(ncomp, h, w, device="cuda", generator=gen) * 2 - 1
    taps = [math.exp(-(t * t) / 128.0) for t in range(-24, 25)]
    for dim in (2, 1):
        size = x.shape[dim]
        at = torch.arange(size, device="cuda")
        y = torch.zeros_like(x)
        for t, k in zip(range(-24, 25), taps):
            y += k * x.index_select(dim, (at + t).clamp(0, size - 1))
        x = y
    x = x * (60.0 / x.abs().amax(dim=(1, 2), keepdim=True)) + 128.0
    return x.round().clamp(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _render(pages, photo):
    """The pages as uint8 arrays (h, w, ncomp) on the GPU."""
    def text(p):
        w, h, ncomp, _, seed = p
        return synth_page(w, h, ncomp, seed).reshape(h, w, ncomp)

    with concurrent.futures.ThreadPoolExecutor(min(16, os.cpu_count() or 1)) as ex:
        sheets = list(ex.map(text, pages))
    out = []
    for (w, h, ncomp, _, seed), sheet in zip(pages, sheets):
        t = torch.from_numpy(sheet).cuda()
        if photo > 0:  # a 4:3 rectangle of that share of the page
            pw = min(w, max(8, int(math.sqrt(photo * w * h * 4 / 3))))
            ph = min(h, max(8, pw * 3 // 4))
            x0, y0 = (seed // 7) % (w - pw + 1), (seed // 11) % (h - ph + 1)
            t[y0:y0 + ph, x0:x0 + pw] = _photo(pw, ph, ncomp, seed)
        out.append(t)
    return out


def _image(page, t):
    make = jl.Image.from_gray_bytes if page[2] == 1 else jl.Image.from_rgb_bytes
    return make(page[0], page[1], t.cpu().numpy().tobytes())


def _format(case, i=0):
    return jl.OutputFormat(case["fmt"] if "fmt" in case else i % 2)


class Room:
    """Where a program keeps a file it has received: a buffer of its own, of a
    length set by the page alone, zero behind the file."""

    def __init__(self, w, h, ncomp, quality):
        samples = w * h * ncomp
        share = 1.0 if samples < 1 << 20 else 0.6 if quality >= 90 else 0.3
        self.buffer = np.zeros(int(samples * share) + 16384, np.uint8)
        self.used = 0

    def keep(self, data):
        n = len(data)
        self.buffer[:n] = np.frombuffer(data, dtype=np.uint8)
        self.buffer[n:self.used] = 0
        self.used = n
        return self.buffer


def prepare(case, seed):
    engine = default_engine()
    pages = _pages(case, seed)
    sheets = _render(pages, case["photo"])
    do = case["do"]
    state = {"do": do, "engine": engine}
    if do != "decode":
        state["rooms"] = [Room(*p[:4]) for p in pages]
    if do == "batch_device":
        torch.cuda.synchronize()
        state["sheets"] = sheets  # keeps the pixels alive
        state["pages"] = [{"px": t.data_ptr(), "on_device": True, "w": p[0], "h": p[1], "ncomp": p[2],
                           "quality": p[3], "fmt": int(_format(case))} for p, t in zip(pages, sheets)]
        return state
    items = [(_image(p, t), jl.EncodeOptions(p[3], _format(case, i)))
             for i, (p, t) in enumerate(zip(pages, sheets))]
    if do == "decode":
        state["files"] = jl.encode_pages(items, engine)
    else:
        state["items"] = items
    return state


def run(state):
    do, engine = state["do"], state["engine"]
    if do == "encode":
        image, options = state["items"][0]
        return state["rooms"][0].keep(jl.encode(image, options, engine))
    if do == "psnr":
        image, options = state["items"][0]
        data, metrics = jl.encode_with_psnr(image, options, engine)
        return {"file": state["rooms"][0].keep(data), "psnr_db": metrics.psnr_db, "ssim": metrics.ssim}
    if do in ("batch", "batch_mixed"):
        files = jl.encode_pages(state["items"], engine)
        return [room.keep(data) for room, data in zip(state["rooms"], files)]
    if do == "batch_device":
        return [room.keep(data) for room, data in zip(state["rooms"], engine.encode_batch(state["pages"]))]
    # lossless colour files and empty code-block segments are the encoder's
    # own output: both flags are what a program that reads them back passes
    if len(state["files"]) == 1:
        return engine.decode(state["files"][0], True, True)[0]
    return [pixels for pixels, _, _, _ in engine.decode_batch(state["files"], True, True)]


def work(case):
    """Pixels on one side, the file (about a bit and a half a sample lossless,
    a third of a bit lossy) on the other; the two-dimensional lifting steps,
    scaling, quantisation and colour transform, about 30 operations a sample."""
    samples = sum(w * h * c for w, h, c, _, _ in _pages(case, 0))
    files = sum(w * h * c * (1.5 if q >= 100 else 0.33) / 8 for w, h, c, q, _ in _pages(case, 0))
    return {"bytes": samples + files, "flops": 30.0 * samples}


def exact(case, seed):
    """Files and samples are whole numbers; the metrics need a decoder, which
    plain numpy is not."""
    return None
