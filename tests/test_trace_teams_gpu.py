"""Ray sets at the sizes where the traversal changes how it deals rays out: one ray per warp, a few
(the lanes of a warp share them), one per lane and one more than that.  Hits must equal the oracle's
bit for bit at every size, for one and several triangles per leaf and for rays of both kinds."""
import numpy as np
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.accel import Accel, set_full_node_leaf, set_max_leaf
from oracle import pyoracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def terrain():
    sc = scenes.large_scene(width=512, height=336, grid=128, n_spheres=40, sky_size=(64, 32))
    tris = sc.world_triangles()
    rays = H.pinhole_rays(sc, jitter_seed=4)
    rng = np.random.default_rng(8)
    rays = rays[rng.permutation(rays.shape[0])]
    rays[::3, 7] = rng.uniform(20, 90, rays[::3].shape[0])     # bounded
    rays[1::5, 3] = rng.uniform(0, 60, rays[1::5].shape[0])    # not from the origin
    mask = (rng.random(tris.shape[0]) < 0.7).astype(np.uint8)
    ob, masked = O.Bvh(tris), O.Bvh(tris)
    masked.set_mask(mask)
    return tris, rays, mask, ob.closest(rays), masked.any(rays)


@pytest.mark.parametrize("leaf", [1, 3])
def test_hits_at_every_way_of_dealing_rays_out(krr_lib, cuda, terrain, leaf):
    tris, rays, mask, want, want_any = terrain
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    try:
        set_max_leaf(leaf)
        set_full_node_leaf(leaf)
        acc = Accel(tris)
    finally:
        set_full_node_leaf(1)
        set_max_leaf(1)
    warps = sms * 8 * 4
    sizes = [1, 2, 3, 4, 5, 31, 32, 33, 127, warps - 1, warps, warps + 1, 3 * warps, 4 * warps + 1,
             5 * warps + 7, 32 * warps, 32 * warps + 1, rays.shape[0]]
    d = torch.from_numpy(rays).cuda()
    for n in (k for k in sizes if k <= rays.shape[0]):
        first = (977 * n) % (rays.shape[0] - n + 1)
        part = d[first:first + n]
        got = acc.trace_closest(part).cpu().numpy()
        assert np.array_equal(got.view(np.uint32), want[first:first + n].view(np.uint32)), n
    acc.set_mask(mask)
    for n in (1, 4, 5, warps, 4 * warps + 1, rays.shape[0]):
        got = acc.trace_any(d[:n]).cpu().numpy()
        assert np.array_equal(got != 0, np.asarray(want_any[:n]) != 0), n
    assert acc.device_errors() == 0
