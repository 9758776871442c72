"""The batched search past the matches that it stages in shared memory (2048) and in
part groups, with 4 to 32 hypotheses per warp: every result of the estimator equals
that of the per-pair call on the same images."""
import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import batch, stages

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pairs(cuda):
    """B is A moved by (17, -9), a part of it replaced: more than 2048 matches, a
    tenth of them wrong; and a small pair beside it."""
    rng = np.random.default_rng(2)
    out = []
    for w, h in ((1000, 900), (300, 240)):
        a = np.kron(rng.integers(0, 256, (h // 4 + 1, w // 4 + 1)), np.ones((4, 4)))[:h, :w]
        a = (0.6 * a + 0.4 * rng.integers(0, 256, (h, w))).astype(np.uint8)
        b = np.roll(a, (-9, 17), (0, 1))
        b[: h // 8] = a[h // 2:h // 2 + h // 8]
        out.append((a, b))
    return out


@pytest.mark.parametrize("hpw", [4, 8, 16, 32])
@pytest.mark.parametrize("hypotheses", [1, 37, 257, 1000, 6000])
def test_many_matches(pairs, hpw, hypotheses):
    knobs = [stages.Knobs(max_keypoints=k, fast_threshold=20, hypotheses=hypotheses, seed=5 + i, levels=2, refinement_steps=2)
             for i, k in enumerate((5000, 400))]
    images = [[torch.from_numpy(g).cuda() for g in p] for p in pairs]
    b = batch.Batch([batch.pair_desc(ia, ib, kn) for (ia, ib), kn in zip(images, knobs)], tuning={"search_hpw": hpw})
    b.enqueue()
    torch.cuda.synchronize()
    runner = stages.PairRunner(1000, 900, 5000, max_r=6000)
    for i, ((ga, gb), kn) in enumerate(zip(pairs, knobs)):
        want, got, out = runner.run(ga, gb, kn), b.result(i), b.outputs(i)
        down = runner.download()
        assert np.array_equal(out["idx_a"], down["idx_a"]) and np.array_equal(out["idx_b"], down["idx_b"])
        assert got["num_matches"] == want["num_matches"] and (i or got["num_matches"] > 2048 + 64)
        for name in ("H", "H_s", "num_inliers", "inlier_ratio", "inlier_coverage", "reproj_residual", "status"):
            assert np.array_equal(got[name], want[name], equal_nan=name in ("H", "H_s", "reproj_residual")), (i, name)
        assert np.array_equal(out["mask"], down["mask"])
