"""The queues as a frame leaves them: nothing in the shadow queue, so that the
stage entry points called after a frame find no ray that it has traced."""
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300._lib import QUEUES
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params", [{"max_depth": 0}, {"max_depth": 1}, {"max_depth": 5}, {"max_depth": 5, "nee": False},
                                    {"max_depth": 5, "levels": 2}, {"max_depth": 5, "wave": 1000}])
def test_no_shadow_rays_left(krr_lib, cuda, params):
    params = dict(params)
    levels, wave = params.pop("levels", 1), params.pop("wave", 0)
    sc = scenes.cornell_box(96, 64)
    pt = WavefrontPathTracer(params)
    pt.set_accel_levels(levels)
    pt.set_launch(wave=wave)
    pt.set_scene(sc)
    pt.resize(96, 64)
    for f in (1, 2):
        pt.begin_frame(f, sc.camera)
        pt.render()
        assert pt.queue_size(QUEUES.index("SHADOW")) == 0
    if not wave:
        before = pt.radiance().clone()
        pt.trace_shadow()
        assert torch.equal(before, pt.radiance())
    assert pt.device_errors() == 0
