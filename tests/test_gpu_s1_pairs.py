"""S1 on pairs whose images take different paths (runs of 48 bytes, four outputs
at a time, the float filter; aligned and odd rows; different working sizes):
each image equals the oracle's, whatever the other one is."""
import ctypes as C
import itertools

import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import _abi
from crossstage_stitch_b200._abi import ImageView, ScaleInfo
from oracle import c_oracle

from .gpu_util import stream

pytestmark = pytest.mark.gpu

# (width, height, pitch alignment of the input, of the output, offset of the output)
SHAPES = [(64, 32, 16, 16, 0), (131, 47, 1, 1, 0), (132, 48, 16, 16, 4), (132, 48, 4, 1, 0), (260, 20, 16, 16, 0), (37, 61, 16, 16, 0)]


def side(rng, w, h, align, out_align, offset, scale):
    rgb = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    pitch = (3 * w + align - 1) // align * align
    rows = torch.zeros((h, pitch), dtype=torch.uint8, device="cuda")
    rows[:, :3 * w] = torch.from_numpy(rgb.reshape(h, 3 * w)).cuda()
    ow, oh = (max(1, int(np.floor(v * scale + 0.5))) for v in (w, h))
    out_pitch = (ow + out_align - 1) // out_align * out_align
    out = torch.full((offset + oh * out_pitch,), 0x5a, dtype=torch.uint8, device="cuda")
    return rgb, rows, out, ImageView(rows.data_ptr(), w, h, pitch, 0), ImageView(out.data_ptr() + offset, ow, oh, out_pitch, 1)


@pytest.mark.parametrize("scale", [1.0, 0.5, 0.25, 0.6])
@pytest.mark.parametrize("a,b", list(itertools.product(range(len(SHAPES)), repeat=2)))
def test_pairs(cuda, scale, a, b):
    rng = np.random.default_rng(10 * a + b)
    sides = [side(rng, *SHAPES[i], scale) for i in (a, b)]
    infos = [ScaleInfo(), ScaleInfo()]
    st = _abi.load().stitch_s1_preprocess(C.byref(sides[0][3]), C.byref(sides[1][3]), scale, C.byref(sides[0][4]),
                                          C.byref(sides[1][4]), C.byref(infos[0]), C.byref(infos[1]), stream())
    torch.cuda.synchronize()
    assert st == 0
    for (rgb, _, out, _, view), i in zip(sides, (a, b)):
        offset = SHAPES[i][4]
        got = out[offset:].view(view.height, view.pitch_bytes).cpu().numpy()
        assert np.array_equal(got[:, :view.width], c_oracle.s1(rgb, view.width, view.height))
        assert (got[:, view.width:] == 0x5a).all() and (out[:offset] == 0x5a).all()
