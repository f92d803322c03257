"""Instance trees of one block's size (up to 1,024 instances) and just above,
built and rebuilt: hits bit-exact against the oracle's two-level restatement,
which tests every instance."""
import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 64, 511, 1023, 1024, 1025])
def test_build_and_update(krr_lib, cuda, n):
    geos, insts = _instanced_scene(seed=n, n_inst=n)
    insts = insts[:n]
    rays = H.random_rays(1500, n, box=5.0)
    acc = Accel.instanced(geos, insts)
    _check(acc, geos, insts, rays, "built")
    for step in (1, 2):
        moved = [(g, np.asarray(m, np.float32).copy()) for g, m in insts]
        for k, (g, m) in enumerate(moved):
            m[:, 3] += np.array([0.4 * np.sin(k + step), 0.3 * step, -0.2 * k / n], np.float32)
        acc.update_instances(np.stack([m for _, m in moved]))
        _check(acc, geos, moved, rays, f"update {step}")


def test_coincident_and_flat_instances(krr_lib, cuda):
    """Equal boxes (equal Morton codes), a flat arrangement and an instance of
    an empty geometry."""
    geos, insts = _instanced_scene(seed=3, n_inst=40)
    geos = list(geos) + [np.zeros((0, 9), np.float32)]
    g0, m0 = insts[0]
    insts = [(g0, m0)] * 30 + [(g, np.asarray(m, np.float32) * np.float32(1)) for g, m in insts[1:20]]
    insts.append((len(geos) - 1, np.asarray(m0, np.float32)))
    acc = Accel.instanced(geos, insts)
    rays = H.random_rays(2000, 4, box=5.0)
    _check(acc, geos, insts, rays, "coincident")
    flat = [(g, np.asarray(m, np.float32).copy()) for g, m in insts]
    for k, (g, m) in enumerate(flat):
        m[:, 3] = (0.1 * k - 2.5, 0.0, 0.0)
    acc.update_instances(np.stack([m for _, m in flat]))
    _check(acc, geos, flat, rays, "in a row")


def test_refused_update_keeps_the_structure(krr_lib, cuda):
    geos, insts = _instanced_scene(seed=8, n_inst=20)
    acc = Accel.instanced(geos, insts)
    rays = H.random_rays(2000, 5, box=5.0)
    xf = np.stack([np.asarray(m, np.float32) for _, m in insts])
    for value in (np.nan, np.inf, -np.inf):
        bad = xf.copy()
        bad[7, 1, 3] = value
        with pytest.raises(Exception):
            acc.update_instances(bad)
        _check(acc, geos, insts, rays, "after a refused update")
    acc.update_instances(xf)
    _check(acc, geos, insts, rays, "updated again")
