"""Instance updates after the process's build settings have changed, and
updates that are refused, below and above the one-block builder's 1,024
instances: hits bit-exact against the oracle's two-level restatement."""
import numpy as np
import pytest
import torch

from kiraray_gb300 import accel as A
from kiraray_gb300.accel import Accel
from oracle import pyoracle as O
from tests import helpers as H
from tests.test_oracle import _instanced_scene

pytestmark = pytest.mark.gpu


def _check(acc, geos, insts, rays, what):
    want = O.trace_instanced(geos, insts, acc.instance_inverse(), rays)
    got = acc.trace_closest(torch.from_numpy(rays).cuda()).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), what
    assert acc.device_errors() == 0


@pytest.mark.parametrize("n", [40, 1030])
@pytest.mark.parametrize("built,now", [(0, 1), (1, 0), (1, 1)])
def test_node_format_set_after_the_build(krr_lib, cuda, n, built, now):
    """Both levels keep the format that the structure was built with."""
    geos, insts = _instanced_scene(seed=n, n_inst=n)
    rays = H.random_rays(2000, n, box=5.0)
    xf = np.stack([np.asarray(m, np.float32) for _, m in insts])
    try:
        A.set_node_format(built)
        acc = Accel.instanced(geos, insts)
        A.set_node_format(now)
        for _ in range(2):
            acc.update_instances(xf)
            _check(acc, geos, insts, rays, "updated")
    finally:
        A.set_node_format(0)


@pytest.mark.parametrize("n", [20, 1025])
def test_refused_update_keeps_the_structure(krr_lib, cuda, n):
    geos, insts = _instanced_scene(seed=8, n_inst=n)
    acc = Accel.instanced(geos, insts)
    rays = H.random_rays(2000, 5, box=5.0)
    xf = np.stack([np.asarray(m, np.float32) for _, m in insts])
    for value in (np.inf, -np.inf):
        bad = xf.copy()
        bad[7, 1, 3] = value
        with pytest.raises(Exception, match="not finite"):
            acc.update_instances(bad)
        _check(acc, geos, insts, rays, "after a refused update")
    with pytest.raises(Exception, match="not finite"):
        acc.update_instances(np.full_like(xf, np.nan))
    _check(acc, geos, insts, rays, "after a refused update")
    acc.update_instances(xf)
    _check(acc, geos, insts, rays, "updated again")
