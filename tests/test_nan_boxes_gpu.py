"""Triangles and instances that are no number anywhere, among others: never
hit, and the others as if they were not there."""
import numpy as np
import pytest
import torch

from kiraray_gb300.accel import Accel
from tests import helpers as H
from tests.test_oracle import _instanced_scene

pytestmark = pytest.mark.gpu


def _hits(acc, rays):
    return acc.trace_closest(torch.from_numpy(rays).cuda()).cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("bad", [1, 40])
def test_triangles(krr_lib, cuda, bad):
    tris = H.random_soup(3000, 5).reshape(-1, 9)
    rays = H.random_rays(20000, 6)
    acc = Accel(np.concatenate([tris, np.full((bad, 9), np.nan, np.float32)]))
    assert np.array_equal(_hits(acc, rays), _hits(Accel(tris), rays))
    assert acc.device_errors() == 0


def test_instances(krr_lib, cuda):
    geos, insts = _instanced_scene(seed=6, n_inst=1200)
    nowhere = np.full((3, 4), np.nan, np.float32)
    rays = H.random_rays(20000, 7, box=5.0)
    acc = Accel.instanced(geos, insts + [(0, nowhere)] * 3)
    assert np.array_equal(_hits(acc, rays), _hits(Accel.instanced(geos, insts), rays))
    assert acc.device_errors() == 0
