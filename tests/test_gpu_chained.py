"""Calls issued one after the other on a stream, whose kernels overlap at their
ends, read what the launch before them wrote: descriptors, layers and matches of
changing images in the same buffers equal those of runs with a wait after every
call."""
import ctypes as C

import numpy as np
import pytest
import torch

from crossstage_stitch_b200 import stages, synth
from crossstage_stitch_b200._abi import ImageView, Matches, S2Config

pytestmark = pytest.mark.gpu
ref = C.byref


class Chain:
    """S2 and S3 of one image (levels > 1: the pyramid call), then S4 against
    fixed descriptors, in the same buffers for every image."""

    def __init__(self, w, h, k, levels, factor):
        self.L, self.w, self.h, self.k = stages.lib(), w, h, k
        dev = torch.device("cuda")
        self.feat, self.fixed = stages.ImageFeatures(k, dev), stages.ImageFeatures(k, dev)
        self.knobs = stages.Knobs(max_keypoints=k, levels=levels, scale_factor=factor)
        self.c2, self.c4, b = S2Config(20, k, 0.04), self.knobs.s4(), C.c_size_t()
        self.ws = []
        for call in ((lambda: self.L.stitch_s2_workspace_bytes(w, h, ref(self.c2), ref(b))),
                     (lambda: self.L.stitch_s3_workspace_bytes(w, h, ref(b))),
                     (lambda: self.L.stitch_pyramid_workspace_bytes(w, h, ref(self.c2), ref(self.knobs.pyramid()), ref(b))),
                     (lambda: self.L.stitch_s4_workspace_bytes(k, k, ref(self.c4), ref(b)))):
            stages.check("workspace_bytes", call())
            self.ws.append((stages.workspace(b.value, dev), b.value))
        self.idx, self.dist = [torch.zeros(k, dtype=torch.int32, device=dev) for _ in range(2)], torch.zeros(k, device=dev)
        self.count = torch.zeros(1, dtype=torch.int32, device=dev)
        self.m = Matches(self.idx[0].data_ptr(), self.idx[1].data_ptr(), self.dist.data_ptr(), k, self.count.data_ptr())

    def features(self, image, feat, wait):
        iv, kp, d, s = ImageView(image.data_ptr(), self.w, self.h, image.stride(0), 1), feat.keypoints(), feat.descriptors(), stages.stream_handle()
        (w2, b2), (w3, b3), (wp, bp), _ = self.ws
        if self.knobs.levels > 1:
            stages.check("pyramid", self.L.stitch_pyramid_detect_describe(
                ref(iv), ref(self.c2), ref(self.knobs.pyramid()), ref(kp), ref(d), stages.ptr(wp), bp, s))
        else:
            stages.check("s2", self.L.stitch_s2_detect(ref(iv), ref(self.c2), ref(kp), stages.ptr(w2), b2, s))
            wait()
            stages.check("s3", self.L.stitch_s3_describe(ref(iv), ref(kp), ref(d), stages.ptr(w3), b3, s))
        wait()

    def match(self, wait):
        args = [x for f in (self.feat, self.fixed) for x in (f.keypoints(), f.descriptors())]
        w4, b4 = self.ws[3]
        stages.check("s4", self.L.stitch_s4_match(*map(ref, args), ref(self.c4), ref(self.m), stages.ptr(w4), b4, stages.stream_handle()))
        wait()
        return [t.clone() for t in (self.feat.count, self.feat.desc, self.count, *self.idx, self.dist)]


@pytest.mark.parametrize("w,h,levels,factor", [(511, 383, 1, 1.2), (511, 383, 4, 1.2), (640, 480, 3, 1.6)])
def test_overlapped_calls(cuda, w, h, levels, factor):
    pair = [synth.make_pair(40 + i, w, h) for i in range(3)]
    images = [torch.from_numpy(g).cuda() for p in pair for g in (p.gray_a, p.gray_b)]
    chain = Chain(w, h, 600, levels, factor)
    chain.features(images[0], chain.fixed, torch.cuda.synchronize)
    want = []
    for im in images:
        chain.features(im, chain.feat, torch.cuda.synchronize)
        want.append([t.cpu().numpy() for t in chain.match(torch.cuda.synchronize)])
    assert int(want[1][2][0]) > 30
    got = []
    for i in range(60):
        chain.features(images[i % 6], chain.feat, lambda: None)
        got.append(chain.match(lambda: None))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        n, m = int(want[i % 6][0][0]), int(want[i % 6][2][0])
        for a, b, rows in zip(g, want[i % 6], (1, n, 1, m, m, m)):
            assert np.array_equal(a.cpu().numpy()[:rows], b[:rows]), i
