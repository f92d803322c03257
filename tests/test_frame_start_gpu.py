"""Frames of as many views as fit a launch's arguments and one more, queued
one after another without a wait; and a training frame captured first."""
import numpy as np
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.nrc import NeuralRadianceCache
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


def _views(n):
    sizes = [(17 + k % 5, 9 + k % 3) for k in range(n)]
    return [(scenes._camera((0.5 + 0.02 * k, 0.5, 0.5 + 1.9), (0.5, 0.5, 0.0), 40.0, w, h), w, h, 7 * k)
            for k, (w, h) in enumerate(sizes)]


@pytest.mark.parametrize("n", [1, 23, 24, 25])
def test_views_by_argument_and_by_copy(krr_lib, cuda, n):
    """Several frames begun before the first is read: each view as its own
    pass renders it, bit for bit."""
    sc = scenes.cornell_box(16, 16)
    views = _views(n)
    pt = WavefrontPathTracer({"max_depth": 4})
    pt.set_scene(sc)
    pt.resize_views(views)
    frames = []
    for f in (1, 2, 3):
        pt.begin_frame_views(f, views)
        frames.append(pt.render_flat().clone())
    frames = [x.cpu().numpy() for x in frames]
    off = 0
    for k, (cam, w, h, seed) in enumerate(views):
        if k in (0, n - 1):
            one = WavefrontPathTracer({"max_depth": 4}, seed=seed)
            one.set_scene(sc)
            one.resize(w, h)
            for f in (1, 2, 3):
                one.begin_frame(f, cam)
                want = one.render().cpu().numpy().reshape(-1, 4)
                assert np.array_equal(frames[f - 1][off:off + w * h].view(np.uint32), want.view(np.uint32)), (k, f)
        off += w * h
    assert pt.device_errors() == 0


def test_training_frame_captured_after_frames_without_training(krr_lib, cuda):
    sc = scenes.cornell_box(64, 48)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        pt = WavefrontPathTracer({"max_depth": 5})
        pt.set_scene(sc)
        pt.resize(64, 48)
        cache = NeuralRadianceCache((0, 0, 0), (1, 1, 1), batch_size=2048)
        out = torch.empty((48, 64, 4), device="cuda")
        pt.set_nrc(cache, train=False)
        pt.begin_frame(1, sc.camera)
        pt.render(out)
        pt.set_nrc(cache, train=True)
        pt.capture_frame(out)
        for f in range(2, 8):
            pt.launch_frame(f)
        s.synchronize()
    assert cache.info().step == 6
    assert torch.isfinite(out).all()
    assert pt.device_errors() == 0
