"""Performance cases of the registration chain, through its public entry points.

listed() names the cases; draw(rng) gives more of the same ranges; prepare()
makes a case's inputs and the handles a program keeps (buffers, plans, captured
graphs, servers); run() is one pass; work() counts what a pass cannot do
without; exact() is the value of computed numbers in 64 bits.

The kinds, and what each stands for in use:

    pair        the drop-in stages on one image pair, S2, S3, S4 and S5 as the
                harness calls them (stages.PairRunner); levels > 1 is the pyramid
    batch       many pairs of one size, one captured graph per step (batch.Batch)
    mixed       one captured batch of pairs of uneven sizes and knobs
    stream      a stream of batches from pinned host buffers (batch.StreamingBatches)
    serve       a burst of host requests through the request loop (server.Server)
    match       S4 alone on two descriptor sets (stitch_s4_match)
    estimate    S5 alone on given matches (stitch_s5_estimate)
    render      S6, the feather panorama of an RGB pair (render.render)
    preprocess  S1, an RGB pair to working-size gray images (stitch_s1_preprocess)

Images follow the recipe of crossstage_stitch_b200.synth (rectangles, blobs and
band-limited noise; view B a noisy homography warp of view A), drawn on the GPU.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from crossstage_stitch_b200 import _abi, batch, render, server, stages, synth
from crossstage_stitch_b200._abi import (Descriptors, HomographyResult, ImageView, Keypoints, Matches, S2Config,
                                         S4Config, S5Config, ScaleInfo)

ref = C.byref


def listed() -> list[dict]:
    return [
        # smallest call: a single-level VGA pair with a small budget, the reference harness's own form
        {"name": "pair_vga_l1", "kind": "pair", "w": 640, "h": 480, "k": 500, "levels": 1, "fast": 20, "r": 500,
         "cross": False},
        # the per-pair configuration of the benchmark: 512x512, 1000 keypoints, 8 levels
        {"name": "pair_512_l8", "kind": "pair", "w": 512, "h": 512, "k": 1000, "levels": 8, "fast": 20, "r": 2000,
         "cross": False},
        # odd sizes, mutual check, a few levels
        {"name": "pair_1279x717_l4", "kind": "pair", "w": 1279, "h": 717, "k": 1999, "levels": 4, "fast": 20,
         "r": 2000, "cross": True},
        # the largest pair: 4K, every knob at its top
        {"name": "pair_4k_l8", "kind": "pair", "w": 3840, "h": 2160, "k": 8000, "levels": 8, "fast": 10, "r": 8000,
         "cross": False},
        # the batched benchmark: 64 pairs of 512x512, images on the device
        {"name": "batch_64x512", "kind": "batch", "n": 64, "w": 512, "h": 512, "k": 2000, "levels": 8, "fast": 20,
         "r": 2000, "cross": False},
        # uneven sizes and knobs in one batch, VGA to 4K
        {"name": "mixed_30", "kind": "mixed", "n": 30, "mix": 1, "levels": 8},
        # the batched benchmark end to end: each step's images come from the host
        {"name": "stream_64x512", "kind": "stream", "n": 64, "w": 512, "h": 512, "k": 2000, "levels": 8, "fast": 20,
         "r": 2000, "cross": False},
        # a burst of uneven host requests to the server, submitted and drained
        {"name": "serve_24", "kind": "serve", "n": 24, "mix": 2, "levels": 8},
        # the matching benchmark: 8192 x 8192 descriptors
        {"name": "match_8192", "kind": "match", "nq": 8192, "nt": 8192, "cross": False},
        # the estimator with every knob at its top: 8000 hypotheses over 8000 matches, half of them wrong
        {"name": "estimate_8000", "kind": "estimate", "m": 8000, "r": 8000, "inliers": 0.5},
        # the panorama of a full-HD pair
        {"name": "render_1080p", "kind": "render", "w": 1920, "h": 1080},
        # a 4K RGB pair to half-size gray
        {"name": "preprocess_4k", "kind": "preprocess", "w": 3840, "h": 2160, "scale": 0.5},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["pair", "pair", "pair", "batch", "batch", "mixed", "stream", "serve", "match", "estimate",
                       "render", "preprocess"])
    fast = rng.choice([10, 20, 40])
    levels = rng.choice([1, 2, 4, 8])
    cross = rng.random() < 0.3
    if kind == "pair":
        w = _log(rng, 300, 3840)
        h = max(240, min(2160, int(w * rng.uniform(0.5, 1.0))))
        return {"kind": kind, "w": w, "h": h, "k": _log(rng, 200, 8000), "levels": levels, "fast": fast,
                "r": _log(rng, 500, 8000), "cross": cross}
    if kind in ("batch", "stream"):
        w = _log(rng, 256, 1280)
        h = max(240, int(w * rng.uniform(0.5, 1.0)))
        n = max(2, min(64, int(16e6 / (w * h)), _log(rng, 4, 64)))
        return {"kind": kind, "n": n, "w": w, "h": h, "k": _log(rng, 300, 2000), "levels": levels, "fast": fast,
                "r": _log(rng, 500, 2000), "cross": cross}
    if kind in ("mixed", "serve"):
        n = _log(rng, 6, 30 if kind == "mixed" else 24)
        return {"kind": kind, "n": n, "mix": rng.randrange(1 << 20), "levels": levels}
    if kind == "match":
        return {"kind": kind, "nq": _log(rng, 200, 8192), "nt": _log(rng, 200, 8192), "cross": cross}
    if kind == "estimate":
        return {"kind": kind, "m": _log(rng, 60, 8000), "r": _log(rng, 500, 8000),
                "inliers": round(rng.uniform(0.3, 0.95), 2)}
    w = _log(rng, 400, 1920 if kind == "render" else 3840)
    h = max(300, int(w * rng.uniform(0.5, 0.75)))
    if kind == "render":
        return {"kind": kind, "w": w, "h": h}
    return {"kind": kind, "w": w, "h": h, "scale": rng.choice([0.25, 0.5, 0.6, 0.75, 1.0])}


# ------------------------------------------------------------------ inputs

DEV = "cuda"


def _scene(g: torch.Generator, rng: random.Random, w: int, h: int) -> torch.Tensor:
    """Rectangles, Gaussian blobs and band-limited noise, clipped to [0, 255]."""
    area = (w * h) / (512.0 * 512.0)
    img = torch.full((h, w), 128.0, dtype=torch.float64, device=DEV)
    for _ in range(max(1, round(60 * area))):
        rw, rh = rng.randrange(8, max(9, w // 6)), rng.randrange(8, max(9, h // 6))
        x0, y0 = rng.randrange(0, max(1, w - rw)), rng.randrange(0, max(1, h - rh))
        img[y0:y0 + rh, x0:x0 + rw] = rng.uniform(0, 255)
    nb = max(1, round(40 * area))
    s = torch.empty(nb, 1, dtype=torch.float64, device=DEV).uniform_(3, 30, generator=g)
    amp = torch.empty(nb, 1, dtype=torch.float64, device=DEV).uniform_(-80, 80, generator=g)
    cx = torch.empty(nb, 1, dtype=torch.float64, device=DEV).uniform_(0, w, generator=g)
    cy = torch.empty(nb, 1, dtype=torch.float64, device=DEV).uniform_(0, h, generator=g)
    xs = torch.arange(w, dtype=torch.float64, device=DEV)
    ys = torch.arange(h, dtype=torch.float64, device=DEV)
    gx = torch.exp(-(xs - cx) ** 2 / (2 * s * s))
    gy = amp * torch.exp(-(ys - cy) ** 2 / (2 * s * s))
    img += gy.T @ gx
    f = torch.fft.rfft2(torch.randn(h, w, dtype=torch.float64, device=DEV, generator=g))
    fy = torch.fft.fftfreq(h, dtype=torch.float64, device=DEV)[:, None]
    fx = torch.fft.rfftfreq(w, dtype=torch.float64, device=DEV)[None, :]
    f[(fx * fx + fy * fy) > 0.01] = 0
    noise = torch.fft.irfft2(f, s=(h, w))
    img += noise * (10.0 / noise.std())
    return img.clamp_(0, 255)


def _warp(src: torch.Tensor, H: np.ndarray) -> torch.Tensor:
    """B(x, y) = A(H [x, y, 1]), bilinear, 0 outside A."""
    h, w = src.shape
    y = torch.arange(h, dtype=torch.float64, device=DEV)[:, None]
    x = torch.arange(w, dtype=torch.float64, device=DEV)[None, :]
    z = H[2, 0] * x + H[2, 1] * y + H[2, 2]
    u = (H[0, 0] * x + H[0, 1] * y + H[0, 2]) / z
    v = (H[1, 0] * x + H[1, 1] * y + H[1, 2]) / z
    inside = (u >= 0) & (v >= 0) & (u <= w - 1) & (v <= h - 1) & (z > 0)
    u, v = torch.where(inside, u, 0.0), torch.where(inside, v, 0.0)
    x0, y0 = u.floor().long(), v.floor().long()
    x1, y1 = (x0 + 1).clamp_(max=w - 1), (y0 + 1).clamp_(max=h - 1)
    fx, fy = u - x0, v - y0
    out = (src[y0, x0] * (1 - fx) * (1 - fy) + src[y0, x1] * fx * (1 - fy) + src[y1, x0] * (1 - fx) * fy +
           src[y1, x1] * fx * fy)
    return torch.where(inside, out, 0.0)


def _pair(seed: int, w: int, h: int, mixed: bool = False):
    """One synthetic pair: (GRAY8 A, GRAY8 B) on the GPU."""
    rng = random.Random(seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    a = _scene(g, rng, w, h)
    H = synth.random_homography(np.random.default_rng(seed), w, h, (0.15, 0.7) if mixed else (0.4, 0.7))
    b = _warp(a, H) + 2.0 * torch.randn(h, w, dtype=torch.float64, device=DEV, generator=g)
    if mixed:  # repeated texture tiles over 20 to 70 % of B
        t = max(16, min(h, w) // 12)
        ty, tx = rng.randrange(0, h - t), rng.randrange(0, w - t)
        tile = b[ty:ty + t, tx:tx + t].clone()
        for _ in range(int(rng.uniform(0.2, 0.7) * (h * w) / (t * t))):
            y, x = rng.randrange(0, h - t), rng.randrange(0, w - t)
            b[y:y + t, x:x + t] = tile
    return [i.round().clamp_(0, 255).to(torch.uint8) for i in (a, b)]


def _knobs(case: dict, seed: int) -> stages.Knobs:
    return stages.Knobs(fast_threshold=case["fast"], max_keypoints=case["k"], hypotheses=case["r"], seed=seed,
                        levels=case["levels"], cross_check=case["cross"])


def _mix(case: dict) -> list[dict]:
    """Sizes and knobs of a mixed batch; they do not depend on the input seed."""
    rng = random.Random(case["mix"])
    out = []
    for i in range(case["n"]):
        w, h = synth.RESOLUTIONS[(i + case["mix"]) % 4]
        out.append({"w": w, "h": h, "k": rng.choice([500, 2000, 8000]), "fast": rng.choice([10, 20, 40]),
                    "r": rng.choice([500, 2000, 8000]), "levels": case["levels"], "cross": False})
    return out


def _result_views(buf: torch.Tensor) -> dict:
    """The numbers of an array of HomographyResult bytes."""
    r = buf.view(-1, C.sizeof(HomographyResult))
    return {"H": r[:, :144].view(torch.float64), "counts": r[:, 144:152].view(torch.int32),
            "measures": r[:, 152:176].view(torch.float64), "status": r[:, 176:180].view(torch.int32)}


def _at(b: batch.Batch, ptr: int, count: int, dtype: torch.dtype) -> torch.Tensor:
    off = ptr - b.ws.data_ptr()
    size = torch.empty(0, dtype=dtype).element_size()
    return b.ws[off:off + count * size].view(dtype)


def _batch_views(b: batch.Batch, i: int) -> dict:
    """Device views of pair i's outputs in a batch's workspace."""
    ka, kb, m = Keypoints(), Keypoints(), Matches()
    da, db = Descriptors(), Descriptors()
    mask, res = C.c_void_p(), C.c_void_p()
    stages.check("pair_outputs", b.lib.stitch_batch_pair_outputs(
        b.plan, C.c_void_p(b.ws.data_ptr()), i, ref(ka), ref(kb), ref(da), ref(db), ref(m), ref(mask), ref(res)))
    k = ka.capacity
    out = {"idx_a": _at(b, m.idx_a, k, torch.int32), "idx_b": _at(b, m.idx_b, k, torch.int32),
           "distance": _at(b, m.distance, k, torch.float32), "matches": _at(b, m.d_count, 1, torch.int32),
           "mask": _at(b, mask.value, k, torch.uint8)}
    for t, kp, d in (("a", ka, da), ("b", kb, db)):
        out |= {"x" + t: _at(b, kp.x, k, torch.float32), "y" + t: _at(b, kp.y, k, torch.float32),
                "r" + t: _at(b, kp.response, k, torch.float32), "n" + t: _at(b, kp.d_count, 1, torch.int32),
                "d" + t: _at(b, d.data, k * 32, torch.uint8)}
    return out


def _uniform_views(b: batch.Batch) -> dict:
    """All outputs of a batch of equal pairs: they lie at equal distances, so
    one strided view holds an output of every pair."""
    first, second, last = _batch_views(b, 0), _batch_views(b, 1), _batch_views(b, b.n - 1)
    whole = b.ws[:b.ws.numel() // 8 * 8]
    out = _result_views(b.results)
    for name, v in first.items():
        size = v.element_size()
        out[name] = whole.view(v.dtype).as_strided((b.n, v.numel()), ((second[name].data_ptr() - v.data_ptr()) // size, 1),
                                                   (v.data_ptr() - b.ws.data_ptr()) // size)
        assert out[name][-1].data_ptr() == last[name].data_ptr()
    return out


def _new_batch(descs) -> batch.Batch:
    b = batch.Batch(descs)
    b.ws.zero_()  # rows past the counts are never written: zero in every run
    torch.cuda.synchronize()
    b.capture()
    return b


def _host(t: torch.Tensor) -> torch.Tensor:
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


# ----------------------------------------------------------------- prepare


def _prepare_pair(case, seed):
    r = stages.PairRunner(case["w"], case["h"], case["k"], max_r=case["r"], cross_check=case["cross"])
    for f in r.feat:  # rows past the counts are never written: zero in every run
        for t in (f.x, f.y, f.response, f.desc):
            t.zero_()
    for t in (r.idx_a, r.idx_b, r.dist):
        t.zero_()
    return {"runner": r, "images": _pair(seed, case["w"], case["h"]), "knobs": _knobs(case, seed)}


def _prepare_batch(case, seed):
    imgs = [_pair(seed * 1000 + i, case["w"], case["h"]) for i in range(case["n"])]
    b = _new_batch([batch.pair_desc(a, bb, _knobs(case, seed + i)) for i, (a, bb) in enumerate(imgs)])
    return {"images": imgs, "batch": b, "out": _uniform_views(b)}


def _prepare_mixed(case, seed):
    mix = _mix(case)
    imgs = [_pair(seed * 1000 + i, c["w"], c["h"], True) for i, c in enumerate(mix)]
    b = _new_batch([batch.pair_desc(a, bb, _knobs(c, seed + i)) for i, (c, (a, bb)) in enumerate(zip(mix, imgs))])
    views = [_batch_views(b, i) for i in range(case["n"])]
    return {"images": imgs, "batch": b,
            "out": {"masks": [v["mask"] for v in views], "da": [v["da"] for v in views]} | _result_views(b.results)}


def _prepare_stream(case, seed):
    sb = batch.StreamingBatches([(case["w"], case["h"], case["w"], case["h"])] * case["n"],
                                [_knobs(case, seed + i) for i in range(case["n"])])
    host = sb.host_buffer()
    for i in range(case["n"]):
        a, b = _pair(seed * 1000 + i, case["w"], case["h"])
        sb.fill(host, i, a.cpu().numpy(), b.cpu().numpy())
    torch.cuda.synchronize()
    for b in sb.batches:  # rows past the counts are never written: zero in every run
        b.ws.zero_()
    return {"sb": sb, "host": host, "prev": None, "out": [_uniform_views(b) for b in sb.batches]}


def _prepare_serve(case, seed):
    mix = _mix(case)
    imgs = [[_host(t) for t in _pair(seed * 1000 + i, c["w"], c["h"], True)] for i, c in enumerate(mix)]
    return {"server": server.Server(arena_bytes=8 << 30), "images": imgs,
            "knobs": [_knobs(c, seed + i) for i, c in enumerate(mix)]}


def _prepare_match(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    nq, nt = case["nq"], case["nt"]
    q = torch.randint(0, 256, (nq, 32), dtype=torch.uint8, device=DEV, generator=g)
    t = torch.randint(0, 256, (nt, 32), dtype=torch.uint8, device=DEV, generator=g)
    # 30 % of the queries get a partner with 5 % of its bits flipped, 5 % a second one at the same distance
    n = max(1, int(0.3 * min(nq, nt)))
    qi = torch.randperm(nq, device=DEV, generator=g)[:n]
    ti = torch.randperm(nt, device=DEV, generator=g)
    for part, rows in ((qi, ti[:n]), (qi[:n // 6], ti[n:n + n // 6])):
        flips = torch.rand(len(part), 32, 8, device=DEV, generator=g) < 0.05
        bits = (flips.to(torch.int32) << torch.arange(8, dtype=torch.int32, device=DEV)).sum(-1).to(torch.uint8)
        t[rows] = q[part][:len(rows)] ^ bits[:len(rows)]
    s = {"q": q, "t": t, "nq": torch.tensor([nq], dtype=torch.int32, device=DEV),
         "nt": torch.tensor([nt], dtype=torch.int32, device=DEV)}
    for name, dtype in (("idx_a", torch.int32), ("idx_b", torch.int32), ("distance", torch.float32)):
        s[name] = torch.zeros(nq, dtype=dtype, device=DEV)
    s["matches"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    cfg = S4Config()
    cfg.ratio_threshold, cfg.cross_check = 0.8, 1 if case["cross"] else 0
    nbytes = C.c_size_t()
    stages.check("s4_workspace_bytes", stages.lib().stitch_s4_workspace_bytes(nq, nt, ref(cfg), ref(nbytes)))
    s["ws"] = stages.workspace(nbytes.value, DEV)
    s["args"] = (Keypoints(0, 0, 0, nq, s["nq"].data_ptr()), Descriptors(0, 32, 32, q.data_ptr()),
                 Keypoints(0, 0, 0, nt, s["nt"].data_ptr()), Descriptors(0, 32, 32, t.data_ptr()), cfg,
                 Matches(s["idx_a"].data_ptr(), s["idx_b"].data_ptr(), s["distance"].data_ptr(), nq,
                         s["matches"].data_ptr()))
    s["bytes"] = nbytes.value
    return s


def _prepare_estimate(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    m, w, h = case["m"], 1920, 1080
    H = torch.tensor(synth.random_homography(np.random.default_rng(seed), w, h, (0.4, 0.7)), device=DEV)
    b = torch.rand(m, 2, dtype=torch.float64, device=DEV, generator=g) * torch.tensor([w - 1, h - 1], device=DEV)
    p = torch.cat([b, torch.ones(m, 1, dtype=torch.float64, device=DEV)], 1) @ H.T
    a = p[:, :2] / p[:, 2:] + 0.7 * torch.randn(m, 2, dtype=torch.float64, device=DEV, generator=g)
    wrong = torch.rand(m, device=DEV, generator=g) >= case["inliers"]
    a[wrong] = torch.rand(int(wrong.sum()), 2, dtype=torch.float64, device=DEV, generator=g) * torch.tensor(
        [w - 1.0, h - 1.0], dtype=torch.float64, device=DEV)
    coords = [v.to(torch.float32).contiguous() for v in (a[:, 0], a[:, 1], b[:, 0], b[:, 1])]
    idx = torch.arange(m, dtype=torch.int32, device=DEV)
    count = torch.tensor([m], dtype=torch.int32, device=DEV)
    dist = torch.zeros(m, dtype=torch.float32, device=DEV)
    mask = torch.zeros(m, dtype=torch.uint8, device=DEV)
    pinned = torch.zeros(C.sizeof(HomographyResult), dtype=torch.uint8, pin_memory=True)
    cfg = S5Config(case["r"], 0, 64, 1, 3.0, seed, 1)
    nbytes = C.c_size_t()
    stages.check("s5_workspace_bytes", stages.lib().stitch_s5_workspace_bytes(ref(cfg), ref(nbytes)))
    kp = [Keypoints(coords[2 * i].data_ptr(), coords[2 * i + 1].data_ptr(), 0, m, count.data_ptr()) for i in (0, 1)]
    scale = stages.make_scale_info(w, h)
    return {"keep": (coords, idx, count, dist), "mask": mask, "pinned": pinned,
            "ws": stages.workspace(nbytes.value, DEV), "bytes": nbytes.value,
            "args": (*kp, Matches(idx.data_ptr(), idx.data_ptr(), dist.data_ptr(), m, count.data_ptr()), scale,
                     scale, cfg), "out": {"mask": mask} | _result_views(pinned)}


def _rgb(seed: int, w: int, h: int) -> list[torch.Tensor]:
    """An RGB pair: the gray pair with a tint per channel."""
    tint = torch.tensor([1.0, 0.9, 0.8], device=DEV)
    return [(i[:, :, None] * tint).to(torch.uint8).contiguous() for i in _pair(seed, w, h)]


def _prepare_render(case, seed):
    w, h = case["w"], case["h"]
    H = [[0.98, 0.02, 0.16 * w], [-0.015, 1.01, 0.02 * h], [1e-5, -2e-5, 1.0]]
    geo = render.prepare_geometry(w, h, w, h, H)
    return {"images": _rgb(seed, w, h), "geo": geo,
            "pano": torch.zeros(geo.height, geo.width, 3, dtype=torch.uint8, device=DEV),
            "mask": torch.zeros(geo.height, geo.width, dtype=torch.uint8, device=DEV)}


def _work_size(case) -> tuple[int, int]:
    return tuple(max(1, int(math.floor(v * case["scale"] + 0.5))) for v in (case["w"], case["h"]))


def _prepare_preprocess(case, seed):
    imgs = _rgb(seed, case["w"], case["h"])
    w, h = _work_size(case)
    gray = [torch.zeros(h, w, dtype=torch.uint8, device=DEV) for _ in range(2)]
    return {"images": imgs, "gray": gray, "scale": case["scale"], "info": (ScaleInfo(), ScaleInfo()),
            "views": [render.rgb_view(t) for t in imgs] + [ImageView(t.data_ptr(), w, h, w, _abi.GRAY8) for t in gray]}


def prepare(case: dict, seed: int) -> dict:
    torch.cuda.set_device(0)
    state = globals()["_prepare_" + case["kind"]](case, seed)
    return {"case": case} | state


# --------------------------------------------------------------------- run


def _run_pair(s):
    r, c = s["runner"], s["case"]
    r.enqueue(c["w"], c["h"], c["w"], c["h"], s["knobs"], images=s["images"])
    out = {"idx_a": r.idx_a, "idx_b": r.idx_b, "distance": r.dist, "matches": r.mcount, "mask": r.mask}
    for t, f in zip("ab", r.feat):
        out |= {"x" + t: f.x, "y" + t: f.y, "r" + t: f.response, "n" + t: f.count, "d" + t: f.desc}
    return out | _result_views(r.pinned)


def _run_batch(s):
    s["batch"].launch()
    return s["out"]


_run_mixed = _run_batch


def _run_stream(s):
    slot = s["sb"].step(s["host"])
    if s["prev"] is not None:  # the step before this one, whose results a program reads now
        s["sb"].wait(s["prev"])
    s["prev"] = slot
    return s["out"][slot]


def _run_serve(s):
    srv = s["server"]
    for i, ((a, b), k) in enumerate(zip(s["images"], s["knobs"])):
        stages.check("submit", srv.submit(a, b, k, tag=i))
    res = sorted(srv.drain(), key=lambda r: r["tag"])
    return {"H": np.stack([r["H"] for r in res]), "H_s": np.stack([r["H_s"] for r in res]),
            "counts": np.array([[r["num_matches"], r["num_inliers"], int(r["status"])] for r in res]),
            "measures": np.array([[r["inlier_ratio"], r["inlier_coverage"], r["reproj_residual"]] for r in res])}


def _run_match(s):
    ka, da, kb, db, cfg, m = s["args"]
    stages.check("s4_match", stages.lib().stitch_s4_match(
        ref(ka), ref(da), ref(kb), ref(db), ref(cfg), ref(m), stages.ptr(s["ws"]), s["bytes"],
        stages.stream_handle()))
    return {k: s[k] for k in ("idx_a", "idx_b", "distance", "matches")}


def _run_estimate(s):
    a, b, m, sa, sb, cfg = s["args"]
    stages.check("s5_estimate", stages.lib().stitch_s5_estimate(
        ref(a), ref(b), ref(m), ref(sa), ref(sb), ref(cfg), stages.ptr(s["mask"]),
        C.c_void_p(s["pinned"].data_ptr()), stages.ptr(s["ws"]), s["bytes"], stages.stream_handle()))
    return s["out"]


def _run_render(s):
    pano, mask = render.render(*s["images"], s["geo"], s["pano"], s["mask"])
    return {"panorama": pano, "mask": mask}


def _run_preprocess(s):
    a, b, ga, gb = s["views"]
    ia, ib = s["info"]
    stages.check("s1_preprocess", stages.lib().stitch_s1_preprocess(
        ref(a), ref(b), s["scale"], ref(ga), ref(gb), ref(ia), ref(ib), stages.stream_handle()))
    return s["gray"]


def run(state: dict):
    return globals()["_run_" + state["case"]["kind"]](state)


# -------------------------------------------------------------------- work


def _layer_pixels(w: int, h: int, levels: int) -> int:
    return sum(round(w / 1.2 ** i) * round(h / 1.2 ** i) for i in range(levels))


def _pair_work(c: dict) -> tuple[float, float]:
    """Bytes: both images in, keypoints, descriptors, matches and mask out.
    Operations: 20 per layer pixel (corner test and smoothing), 1500 per
    keypoint (orientation, 512 rotated samples), 512 per descriptor pair and
    25 per (hypothesis, match), with matches for a third of the keypoints."""
    px, k = c["w"] * c["h"], c["k"]
    bytes_ = 2 * px + 2 * 44 * k + 13 * k
    flops = (2 * 20 * _layer_pixels(c["w"], c["h"], c["levels"]) + 2 * 1500 * k +
             (2 if c["cross"] else 1) * 512 * k * k + 25 * c["r"] * k / 3)
    return bytes_, flops


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "pair":
        b, f = _pair_work(case)
    elif kind in ("batch", "stream"):
        b, f = (case["n"] * v for v in _pair_work(case))
    elif kind in ("mixed", "serve"):
        per = [_pair_work(c) for c in _mix(case)]
        b, f = sum(p[0] for p in per), sum(p[1] for p in per)
    elif kind == "match":
        n, t = case["nq"], case["nt"]
        b, f = 32 * (n + t) + 12 * n, 512 * n * t * (2 if case["cross"] else 1)
    elif kind == "estimate":
        b, f = 25 * case["m"], 25 * case["m"] * case["r"]
    elif kind == "render":
        px = case["w"] * case["h"]
        b, f = 6 * px + 4 * 1.2 * px, 1.2 * px * 80  # canvas about 1.2 times one image
    else:
        px, (w, h) = case["w"] * case["h"], _work_size(case)
        b, f = 2 * (3 * px + w * h), 2 * 6 * px
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------- exact


def exact(case: dict, seed: int):
    """Matching has a value beyond the code's own arithmetic: the distances of
    the accepted matches, from 64-bit dot products. Bytes and whole numbers
    have none, and the homography of a search over minimal samples is defined
    by its own 64-bit operations."""
    if case["kind"] != "match":
        return None
    s = _prepare_match(case, seed)
    bit = torch.arange(8, device=DEV, dtype=torch.uint8)
    q, t = (2.0 * ((s[n][:, :, None] >> bit) & 1).flatten(1).to(torch.float64) - 1 for n in "qt")
    d = (256 - q @ t.T) / 2
    first, second = d.topk(2, largest=False).values.T
    best = (d == first[:, None]).to(torch.uint8).argmax(1)
    ok = torch.where(first == 0, second > 0, first < 0.8 * second)
    if case["cross"]:
        back = (d == d.min(0).values[None, :]).to(torch.uint8).argmax(0)
        ok &= back[best] == torch.arange(case["nq"], device=DEV)
    out = torch.zeros(case["nq"], dtype=torch.float64, device=DEV)
    out[:int(ok.sum())] = first[ok]
    return {"idx_a": None, "idx_b": None, "distance": out, "matches": None}
