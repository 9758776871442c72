"""S2/S3 where the selection, the rank sort, the Harris loads, the describe
rounds, the blur, FAST and the resize change path, bit for bit against the
oracle: tie counts around the ranked and the listed ties, candidate counts
around the rank kernel's blocks and tiles, aligned and odd pitches, tile and
band edges, saturated windows."""
import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import batch, stages
from oracle import pyramid, s2s3
from tests import gpu_util as G
from tests.test_gpu_pyramid import run_pyramid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ours(cuda):
    return G.Lib("ours")


def check(ours, gray, thr, k):
    kp, desc, blurred, (st2, st3, n) = G.detect_describe(ours, gray, thr, k)
    want_kp, want_desc = s2s3.detect_and_describe(gray, thr, k)
    assert (st2, st3) == (0, 0) and n == want_kp.shape[0]
    assert np.array_equal(kp, want_kp) and np.array_equal(desc, want_desc)
    return n


def dots(w, h, step):
    """Equal isolated dots: every one a maximum of the same score."""
    g = np.full((h, w), 60, np.uint8)
    g[::step, ::step] = 200
    return g


@pytest.mark.parametrize("w,h,step,k", [(120, 120, 5, 10),       # some ties, ranked
                                        (222, 222, 5, 100),      # 1024 ties, the last that are ranked
                                        (227, 222, 5, 100),      # one column more: radix select of the tie list
                                        (400, 397, 5, 700),
                                        (701, 703, 5, 3000),     # 16384 ties and a little more: the maxima list
                                        (640, 640, 4, 8192)])
def test_ties(ours, w, h, step, k):
    assert check(ours, dots(w, h, step), 20, k) == k


@pytest.mark.parametrize("k", [1, 63, 64, 65, 511, 512, 513, 1025, 6200])
def test_candidate_counts(ours, k):
    rng = np.random.default_rng(k)
    check(ours, rng.integers(0, 256, (331, 350), dtype=np.uint8), 15, k)


@pytest.mark.parametrize("k", [5919, 9472, 9473, 11839, 11840, 18945, 23680])
def test_describe_rounds(ours, k):
    rng = np.random.default_rng(5)
    check(ours, rng.integers(0, 256, (900, 901), dtype=np.uint8), 10, k)


@pytest.mark.parametrize("pad", [0, 1, 2, 4, 16])
def test_pitches(ours, pad, monkeypatch):
    """Word and byte loads of the Harris window and the orientation disc."""
    monkeypatch.setattr(G, "pitched", lambda gray: pitched(gray, pad))
    rng = np.random.default_rng(9)
    check(ours, rng.integers(0, 256, (200, 256), dtype=np.uint8), 20, 400)


pitched = G.pitched


def test_saturated_blur(ours):
    """The largest blur sums: an all-255 image and its edges against black."""
    g = np.full((150, 170), 255, np.uint8)
    g[70:, 90:] = 0
    g[20:30, 20:30] = 0
    _, _, blurred, _ = G.detect_describe(ours, g, 20, 50)
    assert np.array_equal(blurred, s2s3.blur(g)) and blurred.max() == 255


@pytest.mark.parametrize("w,h,factor", [(134, 134, 1.0001), (135, 147, 1.2), (154, 160, 1.2), (155, 163, 1.2),
                                        (257, 199, 1.44), (263, 258, 1.05), (390, 141, 1.2)])
@pytest.mark.parametrize("aligned", [True, False], ids=["pitch16", "pitch-odd"])
def test_layer_edges(ours, w, h, factor, aligned):
    """FAST groups of eight and resize bands at the edges of their tiles
    (64 pixels from the rim of 3, 128 columns, 16 rows), on noise, where every
    pixel of a layer decides about corners: positions, scores and order."""
    rng = np.random.default_rng(w * 1000 + h)
    gray = rng.integers(0, 256, (h, w), dtype=np.uint8)
    st, kp, _ = run_pyramid(gray, 12, 3000, 3, factor, pad=(-w) % 16 + 16 if aligned else None)
    assert st == 0
    assert np.array_equal(kp, pyramid.detect_and_describe(gray, 12, 3000, 3, factor)[0])


@pytest.mark.parametrize("w,h", [(4, 40), (5, 9), (17, 64), (63, 65), (64, 64), (65, 67), (67, 128), (128, 131), (200, 61)])
@pytest.mark.parametrize("pad", [0, 5, 16])
def test_blur_edges(ours, w, h, pad, monkeypatch):
    """The blurred image at its tiles' edges: mirrored columns and rows, part
    tiles, 16-byte and other pitches."""
    monkeypatch.setattr(G, "pitched", lambda gray: pitched(gray, (-w) % 16 + 16 if pad == 16 else pad))
    g = np.random.default_rng(w * h).integers(0, 256, (h, w), dtype=np.uint8)
    _, _, blurred, (st2, st3, _) = G.detect_describe(ours, g, 20, 50)
    assert (st2, st3) == (0, 0) and np.array_equal(blurred, s2s3.blur(g))


@pytest.mark.parametrize("k", [33, 512, 513])
def test_batched_sort_blocks(cuda, k):
    """20 pairs: more jobs than are ranked; 66 and 1024 candidates a job are
    sorted by small blocks, 1026 by large ones."""
    rng = np.random.default_rng(k)
    grays = [rng.integers(0, 256, (150 + i, 170), dtype=np.uint8) for i in range(40)]
    images = [torch.from_numpy(g).cuda() for g in grays]
    b = batch.Batch([batch.pair_desc(images[2 * i], images[2 * i + 1],
                                     stages.Knobs(max_keypoints=k, fast_threshold=10, hypotheses=64, seed=i))
                     for i in range(20)])
    b.enqueue()
    torch.cuda.synchronize()
    for i in range(0, 40, 7):
        got = b.outputs(i // 2)["kp_a" if i % 2 == 0 else "kp_b"]
        want = s2s3.detect_and_describe(grays[i], 10, k)[0]
        assert want.shape[0] == k and np.array_equal(got, want)


def test_batch_of_many_resize_tiles(cuda):
    """Layers resized by tall tiles (two waves of 128 rows at the first resized
    layer; odd sizes, part tiles) equal the per-pair call's."""
    rng = np.random.default_rng(12)
    pairs = [[rng.integers(0, 256, (h, w), dtype=np.uint8) for _ in range(2)] for w, h in ((3841, 2159), (3700, 2301))]
    images = [[torch.from_numpy(g).cuda() for g in p] for p in pairs]
    knobs = stages.Knobs(max_keypoints=1000, fast_threshold=40, hypotheses=64, levels=4, seed=3)
    b = batch.Batch([batch.pair_desc(ia, ib, knobs) for ia, ib in images])
    b.enqueue()
    torch.cuda.synchronize()
    runner = stages.PairRunner(3841, 2301, 1000, max_r=64)
    for i, (ga, gb) in enumerate(pairs):
        runner.run(ga, gb, knobs)
        want, got = runner.download(), b.outputs(i)
        for key in ("kp_a", "kp_b", "desc_a", "desc_b"):
            assert np.array_equal(got[key], want[key]), (i, key)
