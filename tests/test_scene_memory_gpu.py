"""What a scene's vertices take on the device, and that the way they get there
leaves them as they are: 32 bytes each (position, normal, texture coordinates)
whatever their arrays, read by a pass whose stream waits for no other."""
import dataclasses

import numpy as np
import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.wavefront import WavefrontPathTracer

pytestmark = pytest.mark.gpu


def _frame(sc, levels=1):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        pt = WavefrontPathTracer({"max_depth": 5})
        pt.set_accel_levels(levels)
        pt.set_scene(sc)
        pt.resize(96, 64)
        pt.begin_frame(1, sc.camera)
        out = pt.render().cpu().numpy()
        assert pt.device_errors() == 0
    return out, pt


def _with_vertices(sc, mesh, extra, uv):
    """`extra` more vertices that no triangle of the mesh refers to."""
    m = sc.meshes[mesh]
    rng = np.random.default_rng(extra)
    more = rng.random((extra, 3), dtype=np.float32)
    sc.meshes[mesh] = dataclasses.replace(
        m, positions=np.concatenate([m.positions, more]), normals=np.concatenate([m.normals, more]),
        texcoords=rng.random((m.positions.shape[0] + extra, 2), dtype=np.float32) if uv else None)


@pytest.mark.parametrize("uv", [False, True])
def test_bytes_per_vertex(krr_lib, cuda, uv):
    n = 1 << 23
    plain, _ = _frame(scenes.cornell_box(96, 64))
    sc = scenes.cornell_box(96, 64)
    _with_vertices(sc, 0, n, uv)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    pt = WavefrontPathTracer({"max_depth": 5})
    pt.set_scene(sc)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    # two 2 MB pages' rounding for each of the scene's some twenty arrays
    assert used <= 32 * n + 40 * (2 << 20), used / n
    pt.close()
    got, _ = _frame(sc)
    assert np.array_equal(got.view(np.uint32), plain.view(np.uint32))


@pytest.mark.parametrize("levels", [1, 2])
def test_meshes_of_growing_and_shrinking_arrays(krr_lib, cuda, levels):
    """One mesh after another through the same staging memory: frames of the
    scene without the vertices that nothing refers to."""
    plain, _ = _frame(scenes.cornell_box(96, 64), levels)
    sc = scenes.cornell_box(96, 64)
    for mesh, extra in enumerate((1, 300001, 77, 1 << 20, 5, 100003, 2)):
        _with_vertices(sc, mesh, extra, mesh % 2 == 1)
    got, pt = _frame(sc, levels)
    assert np.array_equal(got.view(np.uint32), plain.view(np.uint32))
    with torch.cuda.stream(torch.cuda.Stream()):
        pt.set_scene(scenes.cornell_box(96, 64))   # and again on the same pass
        pt.begin_frame(1, sc.camera)
        assert np.array_equal(pt.render().cpu().numpy().view(np.uint32), plain.view(np.uint32))
