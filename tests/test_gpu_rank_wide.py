"""Top-K by counting in launches sized far above the keys that are there: every
job's keypoints equal the oracle's when the wide slices are full, part filled and
mostly empty, per image, by layers and in batches that mix jobs for the sort with
jobs for the ranking."""
import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import batch, stages
from oracle import pyramid, s2s3
from tests import gpu_util as G
from tests.test_gpu_pyramid import run_pyramid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,thr", [(28416, 5), (28417, 5), (40000, 5), (40000, 130), (300000, 60)])
def test_one_image(cuda, k, thr):
    """Launches of 1776 slices and more: as many keys as candidates, a part, few."""
    gray = np.random.default_rng(k).integers(0, 256, (700, 701), dtype=np.uint8)
    kp, desc, _, status = G.detect_describe(G.Lib("ours"), gray, thr, k)
    want_kp, want_desc = s2s3.detect_and_describe(gray, thr, k)
    assert status == (0, 0, want_kp.shape[0]) and np.array_equal(kp, want_kp) and np.array_equal(desc, want_desc)


def test_layers(cuda):
    gray = np.random.default_rng(3).integers(0, 256, (500, 640), dtype=np.uint8)
    st, kp, _ = run_pyramid(gray, 20, 60000, 4, 1.2)
    assert st == 0 and np.array_equal(kp, pyramid.detect_and_describe(gray, 20, 60000, 4, 1.2)[0])


@pytest.mark.parametrize("levels", [1, 3])
def test_batch(cuda, levels):
    """Jobs of no, few, 16000 and more than 16384 keys behind capacities of 40000."""
    rng = np.random.default_rng(8)
    sizes = [(200, 150), (620, 600), (62, 90), (120, 640)]
    grays = [rng.integers(0, 256, (h, w), dtype=np.uint8) for w, h in sizes] * 4
    grays[4] = np.full_like(grays[4], 9)
    images = [torch.from_numpy(g).cuda() for g in grays]
    b = batch.Batch([batch.pair_desc(images[2 * i], images[2 * i + 1], stages.Knobs(
        max_keypoints=20000, fast_threshold=4, hypotheses=64, seed=i, levels=levels)) for i in range(8)])
    b.enqueue()
    torch.cuda.synchronize()
    seen = set()
    for i in (0, 1, 2, 3, 4, 13):
        got = b.outputs(i // 2)["kp_a" if i % 2 == 0 else "kp_b"]
        want = (s2s3.detect_and_describe(grays[i], 4, 20000) if levels == 1 else
                pyramid.detect_and_describe(grays[i], 4, 20000, levels, 1.2))[0]
        assert np.array_equal(got, want), i
        seen.add(len(want))
    assert min(seen) == 0 and (levels > 1 or max(seen) == 20000)


@pytest.mark.parametrize("pairs,k,thr", [(3, 4000, 5), (3, 4000, 140), (8, 2000, 5), (8, 2000, 140), (4, 20000, 5)])
def test_batch_decides_by_counts(cuda, pairs, k, thr):
    """Capacities that leave ranking or sorting open: many keys (sorted) and few
    (ranked), by a block per slice and by wide slices; jobs past the sort too."""
    rng = np.random.default_rng(pairs)
    grays = [rng.integers(0, 256, (410 + 40 * (i % 4), 620), dtype=np.uint8) for i in range(2 * pairs)]
    images = [torch.from_numpy(g).cuda() for g in grays]
    b = batch.Batch([batch.pair_desc(images[2 * i], images[2 * i + 1], stages.Knobs(
        max_keypoints=k, fast_threshold=thr, hypotheses=64, seed=i, levels=1)) for i in range(pairs)])
    for _ in range(2):  # the counts are summed up anew in every run
        b.enqueue()
    torch.cuda.synchronize()
    for i in (0, 3, 2 * pairs - 1):
        got = b.outputs(i // 2)["kp_a" if i % 2 == 0 else "kp_b"]
        want = s2s3.detect_and_describe(grays[i], thr, k)[0]
        assert np.array_equal(got, want) and (len(want) == min(k, 20000) or thr == 140 or k == 20000), (i, len(want))
