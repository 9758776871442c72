"""The smallest workspaces that the S2, S3 and pyramid calls accept, and a request's
share of a server's arena, stay what they are: programs hold buffers of these sizes
and budgets that just fit (host arithmetic only)."""
import ctypes as C

import pytest

from crossstage_stitch_b200 import _abi, stages
from crossstage_stitch_b200._abi import Request

# (width, height, K, levels, scale factor): bytes of S2, S3, the pyramid call, a served request
SIZES = {
    (640, 480, 500, 1, 1.2): (492936, 307200, 809472, 2496768),
    (512, 512, 1000, 8, 1.2): (422664, 262144, 2548080, 6012928),
    (512, 512, 2000, 8, 1.2): (438536, 262144, 2575728, 6290176),
    (1279, 717, 1999, 4, 1.2): (1631552, 917043, 7668752, 17785088),
    (3840, 2160, 8000, 8, 1.2): (15982024, 8294400, 91449104, 201191936),
    (1920, 1080, 2000, 3, 1.2): (3816424, 2073600, 15160960, 35090944),
    (1920, 1080, 4000, 16, 1.05): (3848424, 2073600, 64726112, 134719744),
    (300, 240, 50, 11, 1.1): (87288, 72000, 1060480, 2515712),
    (2000, 1500, 700, 9, 1.2): (5586488, 3000000, 32967264, 72331520),
    (800, 600, 3000, 7, 1.3): (843752, 480000, 3663424, 9184768),
}


@pytest.mark.parametrize("case", SIZES)
def test_sizes(case):
    w, h, k, levels, factor = case
    L, ref, b = _abi.load(), C.byref, C.c_size_t()
    kn = stages.Knobs(max_keypoints=k, levels=levels, scale_factor=factor)
    c2, pyr, r = kn.s2(), kn.pyramid(), Request()
    r.width_a = r.pitch_a = r.width_b = r.pitch_b = w
    r.height_a = r.height_b = h
    r.host_a = r.host_b = 256
    r.s2, r.s4, r.s5, r.pyramid = c2, kn.s4(), kn.s5(), pyr
    got = []
    for status in (lambda: L.stitch_s2_workspace_bytes(w, h, ref(c2), ref(b)), lambda: L.stitch_s3_workspace_bytes(w, h, ref(b)),
                   lambda: L.stitch_pyramid_workspace_bytes(w, h, ref(c2), ref(pyr), ref(b)),
                   lambda: L.stitch_server_request_bytes(ref(r), ref(b))):
        assert status() == 0
        got.append(b.value)
    assert all(g <= s for g, s in zip(got, SIZES[case])), (got, SIZES[case])
