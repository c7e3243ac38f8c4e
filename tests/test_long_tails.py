"""Celestial frames with rings or procedural surfaces run one iteration before the
finish kernel takes every path left up to 2^18 samples, then two, with such
surfaces three above 2^21: the megakernel's image and the same bits in every run
on either side, in the scene's own view and in a narrow one, where so many paths
outlive the second iteration that the third one has work."""
import numpy as np
import pytest

from stargaze_b200 import workloads as W
from test_wavefront import assert_same_image, render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp", [
    (512, 512, 1), (512, 513, 1),      # 2^18 samples of whole tiles, and one row of tiles more
    (1024, 1024, 2), (1024, 1025, 2),  # 2^21
    (1024, 1024, 4),                   # 2^22
])
@pytest.mark.parametrize("field", [1.0, 0.2])
@pytest.mark.parametrize("styled", [False, True], ids=["rings", "styled"])
def test_long_tails_render_the_megakernel_image(styled, field, width, height, spp):
    wl = W.rings_1080p(width, height)
    wl.frame.globals.cam_forward[3] *= field
    if styled:
        planet = wl.frame.bodies[2]
        planet.axis_x[3], planet.axis_y[3] = 1.0, 17.0
        planet.surface_color[:] = [0.3, 0.27, 0.22, 0.5]
        planet.surface_params[:] = [7.0, 1.0, 0.0, 0.0]
    mega, _, _ = render(wl, "megakernel", 1, spp)
    wave, _, _ = render(wl, "wavefront", 1, spp)
    again, _, _ = render(wl, "wavefront", 1, spp)
    assert np.abs(mega[:, :3]).sum() > 0
    assert np.array_equal(wave, again)
    assert_same_image(wave, mega)
