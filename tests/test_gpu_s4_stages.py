"""The tensor-core matchers where a half stage, a key fold or a column half ends:
train counts around multiples of 32 rows up to several folds, query counts
around a tile, bit for bit against the oracle (ties everywhere: few distinct
descriptors)."""
import numpy as np
import pytest

from crossstage_stitch_b200 import _abi
from tests import gpu_util as G
from tests.test_gpu_s4 import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [1, 2, 3, 4])
@pytest.mark.parametrize("nq,nt", [(1, 1), (127, 31), (128, 33), (129, 64), (130, 127), (64, 128), (200, 129), (128, 255),
                                   (128, 257), (300, 511), (128, 513), (128, 1024), (257, 1025), (128, 2048 + 31)])
def test_half_stages(cuda, kind, nq, nt):
    rng = np.random.default_rng(1000 * nq + nt)
    pool = rng.integers(0, 256, (max(2, nt // 3), 32), dtype=np.uint8)
    pool[0], pool[1] = 0, 255  # distances 0 and 256
    q, t = pool[rng.integers(0, len(pool), nq)], pool[rng.integers(0, len(pool), nt)]
    L = _abi.load()
    before = L.stitch_s4_matcher()
    assert L.stitch_s4_set_matcher(kind) == 0
    try:
        check(G.Lib("ours"), q, t, cross=True, pad_a=0, pad_b=0)
    finally:
        L.stitch_s4_set_matcher(before)
    assert L.stitch_s4_tc_errors() == 0
