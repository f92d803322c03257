"""An instance update on one stream while traces launched before it still run
on another: those see the old transforms, later ones the new."""
import numpy as np
import pytest
import torch

from kiraray_gb300.accel import Accel
from tests import helpers as H
from tests.test_oracle import _instanced_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 1024])
def test_traces_in_flight_on_another_stream(krr_lib, cuda, n):
    geos, insts = _instanced_scene(seed=n, n_inst=n)
    insts = insts[:n]
    there = np.stack([np.asarray(m, np.float32) for _, m in insts])
    away = there.copy()
    away[:, :, 3] += np.float32(3.0)
    acc = Accel.instanced(geos, insts)
    rays = torch.from_numpy(H.random_rays(1 << 20, n, box=5.0)).cuda()
    old = acc.trace_closest(rays).clone()
    acc.update_instances(away)
    new = acc.trace_closest(rays).clone()
    acc.update_instances(there)
    assert not torch.equal(old.view(torch.int32), new.view(torch.int32))
    other = torch.cuda.Stream()
    outs = [torch.empty_like(old) for _ in range(8)]
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(other):
            for o in outs:
                acc.trace_closest(rays, o)
        acc.update_instances(away)
        after = acc.trace_closest(rays)
        acc.update_instances(there)
        torch.cuda.synchronize()
        for o in outs:
            assert torch.equal(o.view(torch.int32), old.view(torch.int32))
        assert torch.equal(after.view(torch.int32), new.view(torch.int32))
    assert acc.device_errors() == 0


@pytest.mark.parametrize("mode", ["thread_local", "global", "relaxed"])
def test_captured_traces_in_flight(krr_lib, cuda, mode):
    """A captured trace runs on whatever stream its graph is launched on."""
    geos, insts = _instanced_scene(seed=7, n_inst=300)
    there = np.stack([np.asarray(m, np.float32) for _, m in insts])
    away = there.copy()
    away[:, :, 3] += np.float32(3.0)
    acc = Accel.instanced(geos, insts)
    rays = torch.from_numpy(H.random_rays(1 << 20, 7, box=5.0)).cuda()
    old = acc.trace_closest(rays).clone()
    outs, beside = [torch.empty_like(old) for _ in range(6)], torch.empty_like(old)
    capturing, other = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(capturing):
        graph.capture_begin(capture_error_mode=mode)
        try:
            for o in outs:
                acc.trace_closest(rays, o)
            with torch.cuda.stream(other):       # an ordinary trace beside the capture
                acc.trace_closest(rays, beside)
        finally:
            graph.capture_end()
    torch.cuda.synchronize()
    assert torch.equal(beside.view(torch.int32), old.view(torch.int32))
    acc.update_instances(away)
    new = acc.trace_closest(rays).clone()
    for _ in range(3):
        acc.update_instances(there)
        with torch.cuda.stream(other):
            graph.replay()
        acc.update_instances(away)
        after = acc.trace_closest(rays)
        torch.cuda.synchronize()
        for o in outs:
            assert torch.equal(o.view(torch.int32), old.view(torch.int32))
        assert torch.equal(after.view(torch.int32), new.view(torch.int32))
    assert acc.device_errors() == 0


def test_frames_in_flight_on_another_stream(krr_lib, cuda):
    """A pass's frame with media reads the instance tree in its own kernels
    too; its structure traced meanwhile on another stream, through the pass's
    accelerator."""
    from kiraray_gb300 import scenes
    from kiraray_gb300.wavefront import WavefrontPathTracer
    sc = scenes.volume_box(256, 192, max_depth=6, grid=32)
    k = len(sc.instances) - 1
    moved = np.asarray(sc.instances[k][1], np.float32).copy()
    moved[0, 3] += np.float32(0.05)

    def fresh(xf):
        other = scenes.volume_box(256, 192, max_depth=6, grid=32)
        other.instances[k] = (other.instances[k][0], xf)
        pt = WavefrontPathTracer({"max_depth": 6})
        pt.set_accel_levels(2)
        pt.set_scene(other)
        pt.resize(256, 192)
        pt.begin_frame(1, other.camera)
        return pt.render().clone()

    want = [fresh(sc.instances[k][1]), fresh(moved)]
    pt = WavefrontPathTracer({"max_depth": 6})
    pt.set_accel_levels(2)
    pt.set_scene(sc)
    pt.resize(256, 192)
    for i in range(4):
        pt.update_instances([k], np.asarray(moved if i % 2 else sc.instances[k][1], np.float32)[None])
        pt.begin_frame(1, sc.camera)
        assert torch.equal(pt.render(), want[i % 2])
    assert pt.device_errors() == 0
