"""S1's integer modes through their 8-byte, 4-byte, shifted and byte loads, and
its word and byte stores: every alignment of the source and of the output, odd
widths, the image's first and last bytes, against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import _abi
from crossstage_stitch_b200._abi import ImageView, ScaleInfo
from oracle import c_oracle

from .gpu_util import stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factor", [1, 2, 4])
@pytest.mark.parametrize("w,h", [(4, 1), (5, 3), (64, 9), (131, 17), (257, 6)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (0, 8), (0, 4), (1, 0), (2, 5), (3, 1), (4, 4), (7, 3)])
def test_loads(cuda, factor, w, h, offset, pad):
    rng = np.random.default_rng(w * 100 + h + offset)
    sw, sh = w * factor, h * factor
    rgb = rng.integers(0, 256, (sh, sw, 3), dtype=np.uint8)
    pitch = 3 * sw + pad
    buf = torch.zeros(offset + sh * pitch, dtype=torch.uint8, device="cuda")
    rows = buf[offset:offset + sh * pitch].view(sh, pitch)
    rows[:, :3 * sw] = torch.from_numpy(rgb.reshape(sh, 3 * sw)).cuda()
    out_pitch = w + pad
    out = torch.full((offset + h * out_pitch,), 0x5a, dtype=torch.uint8, device="cuda")
    si = ScaleInfo()
    st = _abi.load().stitch_s1_preprocess_single(
        C.byref(ImageView(buf.data_ptr() + offset, sw, sh, pitch, 0)), 1.0 / factor,
        C.byref(ImageView(out.data_ptr() + offset, w, h, out_pitch, 1)), C.byref(si), stream())
    torch.cuda.synchronize()
    assert st == 0
    got = out[offset:].view(h, out_pitch).cpu().numpy()
    assert np.array_equal(got[:, :w], c_oracle.s1(rgb, w, h))
    assert (got[:, w:] == 0x5a).all() and (out[:offset] == 0x5a).all()


@pytest.mark.parametrize("factor", [1, 2, 4])
@pytest.mark.parametrize("w,h", [(15, 2), (16, 17), (20, 5), (37, 33), (263, 6)])
@pytest.mark.parametrize("out_offset", [0, 4, 8])
def test_runs(cuda, factor, w, h, out_offset):
    """48-byte runs of 16-byte aligned rows and their last, shorter one; an
    output that the run's store does not fit."""
    rng = np.random.default_rng(w + h)
    sw, sh = w * factor, h * factor
    rgb = rng.integers(0, 256, (sh, sw, 3), dtype=np.uint8)
    pitch, out_pitch = (3 * sw + 15) // 16 * 16, (w + 15) // 16 * 16
    rows = torch.zeros((sh, pitch), dtype=torch.uint8, device="cuda")
    rows[:, :3 * sw] = torch.from_numpy(rgb.reshape(sh, 3 * sw)).cuda()
    out = torch.full((out_offset + h * out_pitch,), 0x5a, dtype=torch.uint8, device="cuda")
    si = ScaleInfo()
    st = _abi.load().stitch_s1_preprocess_single(
        C.byref(ImageView(rows.data_ptr(), sw, sh, pitch, 0)), 1.0 / factor,
        C.byref(ImageView(out.data_ptr() + out_offset, w, h, out_pitch, 1)), C.byref(si), stream())
    torch.cuda.synchronize()
    assert st == 0
    got = out[out_offset:].view(h, out_pitch).cpu().numpy()
    assert np.array_equal(got[:, :w], c_oracle.s1(rgb, w, h))
    assert (got[:, w:] == 0x5a).all() and (out[:out_offset] == 0x5a).all()
