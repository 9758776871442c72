"""S5 at the match counts where its kernels change path: the edges of the
16-term groups, of the loss and normal-matrix chunks and of the points staged
in shared memory, bit for bit against the oracle."""
import numpy as np
import pytest

from tests import gpu_util as G
from tests.test_gpu_s5 import oracle_s5, synthetic_matches

pytestmark = pytest.mark.gpu


def check(n, frac, R, refine, seed, tau=3.0, scale=1.0):
    f = G.S5Fixture(G.Lib("ours"), n)
    a, b_orig, ia, perm, b = synthetic_matches(seed, n, frac)
    a, b = (a * np.float32(scale)).astype(np.float32), (b * np.float32(scale)).astype(np.float32)
    inv = np.argsort(perm)
    f.set_points(a, b, ia, inv)
    f.config.hypotheses, f.config.threshold, f.config.seed, f.config.refinement_steps = R, tau, seed * 31, refine
    got = f.run()
    want, wmask, _ = oracle_s5(f, a, b, ia, inv, R, tau, seed * 31, refine)
    assert got["status"] == want["status"] and got["num_inliers"] == want["num_inliers"]
    assert np.array_equal(f.mask_host()[:n], wmask[:n])
    if want["status"] == 0:
        for name in ("H_s", "H"):
            assert np.array_equal(got[name], want[name].reshape(9))
        for name in ("inlier_ratio", "reproj_residual", "inlier_coverage"):
            assert got[name] == want[name]


@pytest.mark.parametrize("n", [15, 16, 17, 112, 113, 447, 449, 465, 897, 8192, 8193, 8300])
def test_match_counts(cuda, n):
    check(n, 0.0 if n < 20 else 0.3, 64, 2, seed=n)


@pytest.mark.parametrize("R", [1, 7, 9, 1184, 1185, 2369, 4737, 9600])
def test_hypothesis_counts(cuda, R):
    """8, 16, 32 and 64 hypotheses per block, partial groups, several groups per block."""
    check(97, 0.4, R, 1, seed=R)


@pytest.mark.parametrize("tau,scale", [(1e-7, 1.0), (0.05, 1.0), (2e6, 1.0), (3.0, 3000.0), (500.0, 1e-3), (1e-3, 1e-6)])
def test_bounds_range(cuda, tau, scale):
    """Thresholds and coordinates inside and outside the range of the FP32
    bounds, and thresholds that every or no match meets."""
    check(301, 0.3, 700, 1, seed=77, tau=tau, scale=scale)
