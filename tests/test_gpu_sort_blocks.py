"""The batched sort by blocks of 256, 512 and 1024 threads: candidate counts at the
edges between them, against the oracle."""
import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import batch, stages
from oracle import s2s3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,k", [(24, 256), (24, 257), (24, 512), (24, 513), (450, 300)])
def test_blocks(cuda, pairs, k):
    """48 jobs: 512 candidates and fewer by 256 threads, 514 and 1024 by 512, 1026 by
    1024; 900 jobs of 600 by 256 again."""
    rng = np.random.default_rng(k)
    grays = [rng.integers(0, 256, (150 + i, 170), dtype=np.uint8) for i in range(6)]
    images = [torch.from_numpy(g).cuda() for g in grays]
    b = batch.Batch([batch.pair_desc(images[i % 6], images[(i + 1) % 6], stages.Knobs(
        max_keypoints=k, fast_threshold=10, hypotheses=32, seed=i)) for i in range(pairs)])
    b.enqueue()
    torch.cuda.synchronize()
    want = [s2s3.detect_and_describe(g, 10, k)[0] for g in grays]
    for i in (0, 1, 5, pairs // 2, pairs - 1):
        out = b.outputs(i)
        assert np.array_equal(out["kp_a"], want[i % 6]) and np.array_equal(out["kp_b"], want[(i + 1) % 6]) and len(out["kp_a"]) == k
