"""Descriptors where far fewer keypoints are there than the capacities allow for:
the describe blocks take fewer keypoints each, per image, by layers and in batches,
with every keypoint described once."""
import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import batch, stages
from oracle import pyramid, s2s3
from tests import gpu_util as G
from tests.test_gpu_pyramid import run_pyramid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,thr", [(11840, 120), (23680, 100), (23680, 60), (47360, 140), (47360, 60), (200000, 100), (200000, 20)])
def test_one_image(cuda, k, thr):
    """16, 32 and 64 keypoints per block by the capacity; some hundred to some ten
    thousand there."""
    gray = np.random.default_rng(thr).integers(0, 256, (600, 641), dtype=np.uint8)
    kp, desc, _, status = G.detect_describe(G.Lib("ours"), gray, thr, k)
    want_kp, want_desc = s2s3.detect_and_describe(gray, thr, k)
    assert status == (0, 0, want_kp.shape[0]) and 0 < len(want_kp) < k
    assert np.array_equal(kp, want_kp) and np.array_equal(desc, want_desc)


@pytest.mark.parametrize("thr", [15, 60])
def test_layers(cuda, thr):
    """Smooth texture, on which the fused sums of the layers' blur agree with the oracle's."""
    rng = np.random.default_rng(thr)
    coarse = rng.integers(0, 256, (100, 130)).astype(np.uint8)
    gray = np.kron(coarse, np.ones((5, 5), np.uint8))
    st, kp, desc = run_pyramid(gray, thr, 60000, 3, 1.2)
    want_kp, want_desc = pyramid.detect_and_describe(gray, thr, 60000, 3, 1.2)
    assert st == 0 and len(want_kp) > 500 and np.array_equal(kp, want_kp)
    assert (desc == want_desc).mean() > 0.9999


def test_batch_equals_full_capacity(cuda):
    """The same images with a capacity that the keypoints fill and with one that they
    do not."""
    rng = np.random.default_rng(4)
    images = [torch.from_numpy(np.kron(rng.integers(0, 256, (60, 70)), np.ones((5, 5))).astype(np.uint8)).cuda() for _ in range(8)]

    def run(k):
        b = batch.Batch([batch.pair_desc(images[2 * i], images[2 * i + 1], stages.Knobs(
            max_keypoints=k, fast_threshold=30, hypotheses=64, seed=i, levels=1)) for i in range(4)])
        b.enqueue()
        torch.cuda.synchronize()
        return [b.outputs(i) for i in range(4)]
    many = run(30000)
    for i, out in enumerate(many):
        n = max(len(out["kp_a"]), len(out["kp_b"]))
        assert 300 < n < 10000
        few = run(n)[i]
        for key in ("kp_a", "kp_b", "desc_a", "desc_b"):
            assert np.array_equal(out[key], few[key]), (i, key)
