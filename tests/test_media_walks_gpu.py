"""The majorant walks over scalar and coloured spectra, and tracking launches
with fewer items than lanes, warps or a warp's share, against the CPU
restatement (tolerance of tests/test_wavefront_gpu.py)."""
import numpy as np
import pytest

from kiraray_gb300 import scenes
from kiraray_gb300.wavefront import WavefrontPathTracer
from oracle import pyoracle as O
from tests.test_wavefront_gpu import compare, gpu_frame

pytestmark = pytest.mark.gpu


def _volume(w, h, sigma_t, albedo):
    sc = scenes.volume_box(w, h, max_depth=8, grid=32)
    m = sc.media[0]
    sc.media[0] = scenes.Medium(m.density, m.bounds_min, m.bounds_max, sigma_t=sigma_t, albedo=albedo, g=0.3,
                                scale=20.0, majorant_res=(16, 16, 16))
    return sc


@pytest.mark.parametrize("sigma_t,albedo", [((1, 1, 1), (0.9, 0.9, 0.9)), ((1.0, 0.6, 0.3), (0.9, 0.9, 0.9)),
                                            ((1, 1, 1), (0.9, 0.8, 0.95)), ((1, 1, 0.0), (0.9, 0.9, 0.9))])
def test_grey_and_coloured_grid(krr_lib, cuda, sigma_t, albedo):
    sc = _volume(96, 80, sigma_t, albedo)
    pt = WavefrontPathTracer({"max_depth": 8})
    pt.set_scene(sc)
    pt.resize(sc.width, sc.height)
    L, _ = gpu_frame(pt, sc, 2)
    assert pt.device_errors() == 0
    oL, _ = O.PathTracer(sc).render({"max_depth": 8}, 2)
    compare(L[:, :3], oL, f"sigma_t {sigma_t}, albedo {albedo}")


@pytest.mark.parametrize("block", [64, 256])
def test_any_number_of_items(krr_lib, cuda, block):
    """A path depends on its pixel alone: the same frame whatever the waves
    that it is rendered in, from one item a launch to more than the resident
    lanes take at once, and again on the same pass."""
    sc = _volume(400, 300, (1, 1, 1), (0.9, 0.9, 0.9))
    frames = []
    for wave in (0, 0, 33, 4097, 77777):
        pt = WavefrontPathTracer({"max_depth": 3 if wave == 33 else 8})
        pt.set_launch(block=block, wave=wave)
        pt.set_scene(sc)
        if wave == 33:      # a corner of the frame in many small waves
            cam = scenes.cornell_box(24, 16).camera
            pt.resize(24, 16)
            pt.begin_frame(1, cam)
            small = pt.render().cpu().numpy()
            whole = WavefrontPathTracer({"max_depth": 3})
            whole.set_scene(sc)
            whole.resize(24, 16)
            whole.begin_frame(1, cam)
            assert np.array_equal(small, whole.render().cpu().numpy())
            continue
        pt.resize(sc.width, sc.height)
        for _ in range(2):
            pt.begin_frame(1, sc.camera)
            frames.append(pt.render().cpu().numpy())
        assert pt.device_errors() == 0
    for f in frames[1:]:
        assert np.array_equal(frames[0], f)
