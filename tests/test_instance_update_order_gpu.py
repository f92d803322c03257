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
