"""Scatter launches with one thread per item and with two (light sample and
BSDF sample by different warps): the same frame, bit for bit, as one thread
per path computes (the megakernel)."""
import numpy as np
import pytest

from kiraray_gb300 import scenes
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,block", [(1, 1, 256), (33, 1, 64), (63, 65, 128), (241, 135, 256), (256, 228, 256),
                                       (257, 228, 256), (480, 270, 64)])
def test_frame_equals_the_megakernel(krr_lib, cuda, w, h, block):
    sc = scenes.large_scene(w, h, grid=65, n_spheres=60)
    for nee in (True, False):
        pt = WavefrontPathTracer({"max_depth": 6, "nee": nee})
        pt.set_launch(block=block)
        pt.set_scene(sc)
        pt.resize(w, h)
        for frame in (1, 2):
            pt.begin_frame(frame, sc.camera)
            a = pt.render().cpu().numpy()
            pt.begin_frame(frame, sc.camera)
            b = pt.render_megakernel().cpu().numpy()
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (nee, frame)
        assert pt.device_errors() == 0
