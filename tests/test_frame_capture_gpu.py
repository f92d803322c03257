"""Beginning a frame on a stream that is being captured is refused: a replay
would render that frame's index and cameras again, whatever frame is asked for."""
import numpy as np
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 24, 25])
def test_begin_frame_in_a_capture_is_refused(krr_lib, cuda, n):
    sc = scenes.cornell_box(16, 12)
    views = [(sc.camera, 16, 12, k) for k in range(n)]
    pt = WavefrontPathTracer({"max_depth": 3})
    pt.set_scene(sc)
    pt.resize_views(views)
    pt.begin_frame_views(1, views)
    want = pt.render_flat().clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            with pytest.raises(Exception, match="captur"):
                pt.begin_frame_views(2, views)
        finally:
            graph.capture_end()
    torch.cuda.synchronize()
    pt.begin_frame_views(1, views)
    assert np.array_equal(pt.render_flat().cpu().numpy(), want.cpu().numpy())
    assert pt.device_errors() == 0
