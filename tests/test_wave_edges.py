"""The wavefront where its bookkeeping has edges. A dispatch larger than the pool
lists the tiles to trace in raster order, 1024 at a time: more of them than that,
against the same scene traced without a list (padded past 32 bodies). Images
smaller than a tile, or of a tile and a remainder, against the megakernel. Compared
pixel by pixel with a bar of 1e-3: shading rounds differently by ulps, a tile or a
sample that is lost or counted twice shows as a fraction of the pixel."""
import numpy as np
import pytest

from stargaze_b200 import workloads as W
from stargaze_b200.pathtracer import PathTracer
from stargaze_b200.scene import body
from test_camera_tiles import scene
from test_wavefront import render, small_terrain

pytestmark = pytest.mark.gpu


def assert_every_pixel(a, b):
    np.testing.assert_array_equal(a[:, 3], b[:, 3])
    np.testing.assert_array_equal(a[:, :3] > 0, b[:, :3] > 0)
    np.testing.assert_allclose(a[:, :3], b[:, :3], rtol=1e-3, atol=0)


@pytest.mark.parametrize("seed", range(4))
def test_raster_list_of_more_tiles_than_a_round(seed):
    width, height = 1001, 563  # 63 x 36 tiles
    images = []
    for padded in (False, True):
        f = scene(seed, width, height)
        if padded:
            f.bodies += [body([0.0, 0.0, 5.0 + k], 0.0, [0.0] * 3, False) for k in range(33 - len(f.bodies))]
        wl = W.Workload("tiles", f, width, height, 2, 1, {}, "")
        t = PathTracer((width, height), W.render_options(wl, 2, noise_seed=seed))
        t.set_integrator("wavefront", 1 << 16)
        t.encode(f)
        images.append(t.read_pixels())
        t.close()
    assert np.isfinite(images[0]).all()
    assert_every_pixel(*images)


@pytest.mark.parametrize("name", ["rings", "terrain"])
def test_small_images_render_the_megakernels(name):
    lit = 0.0
    for width, height, spp in [(1, 1, 1), (16, 16, 1), (17, 15, 3)]:
        wl = W.rings_1080p(width, height) if name == "rings" else small_terrain(width, height)
        mega, _, _ = render(wl, "megakernel", 2, spp)
        wave, _, _ = render(wl, "wavefront", 2, spp)
        assert_every_pixel(wave, mega)
        lit += float(np.abs(mega[:, :3]).sum())
    assert lit > 0
