"""Captured frames of a pass with two levels and instance updates: replayed
with the moved instances while the instance tree stays in place, dropped when
it moves to new buffers."""
import numpy as np
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


def _pass(sc):
    pt = WavefrontPathTracer({"max_depth": 3})
    pt.set_accel_levels(2)
    pt.set_scene(sc)
    pt.resize(sc.width, sc.height)
    return pt


@pytest.mark.parametrize("n", [20, 1100])
def test_replay_after_update(krr_lib, cuda, n):
    sc = scenes.large_scene(64, 48, grid=33, n_spheres=n, sphere_level=1)
    # one sphere's mesh for all (a structure holds up to 255 geometries)
    sc.instances = [(1 if 1 <= m <= n else m, xf) for m, xf in sc.instances]
    assert (len(sc.instances) > 1024) == (n > 1024)
    index = list(range(1, 11))
    xf = np.stack([np.asarray(sc.instances[k][1], np.float32) for k in index])
    xf[:, 1, 3] += np.float32(4.0)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        pt = _pass(sc)
        out = torch.empty((48, 64, 4), device="cuda")
        pt.begin_frame(1, sc.camera)
        pt.render(out)
        pt.capture_frame(out)
        pt.update_instances(index, xf)
        if n > 1024:
            with pytest.raises(Exception, match="capture"):
                pt.launch_frame(2)
            pt.capture_frame(out)
        pt.launch_frame(2)
        s.synchronize()
        got = out.cpu().numpy()
        for k, m in zip(index, xf):
            sc.instances[k] = (sc.instances[k][0], m)
        fresh = _pass(sc)
        fresh.begin_frame(2, sc.camera)
        want = fresh.render().cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert pt.device_errors() == 0
