"""Rays exactly through shared vertices and edges, from both sides and along each axis: zero
barycentrics must carry the oracle's sign, whichever way the ray crosses the triangle's winding."""
import numpy as np
import pytest
import torch

from kiraray_gb300.accel import Accel
from oracle import pyoracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [1, -1])
@pytest.mark.parametrize("flip", [False, True])
def test_zero_barycentrics_through_edges(krr_lib, cuda, axis, side, flip):
    tris = H.grid_mesh(8).reshape(-1, 3, 3)
    rays = H.vertex_edge_rays(8, 3)
    straight = rays.copy()          # onto the same points along the axis: exact cancellations
    straight[:, :3] += straight[:, 4:7]
    straight[:, 2] = 1.0
    straight[:, 4:7] = (0.0, 0.0, -1.0)
    rays = np.concatenate([rays, straight])
    rays[:, 2] *= side
    rays[:, 6] *= side
    order = np.roll([0, 1, 2], axis)
    tris = np.ascontiguousarray(tris[:, ::-1] if flip else tris)[:, :, order].reshape(-1, 9).copy()
    rays[:, :3], rays[:, 4:7] = rays[:, :3][:, order], rays[:, 4:7][:, order]
    got = Accel(tris).trace_closest(torch.from_numpy(rays).cuda()).cpu().numpy()
    want = O.closest_brute(tris, rays)
    assert (want[:, 1:3] == 0).any()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
