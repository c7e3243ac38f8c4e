"""Dispatches the host enqueues without asking the GPU (one or two stage
iterations, then the finish kernel for every path left) and the ones it follows:
the same image as the per-pixel megakernel at the sizes where the rule changes
(samples per dispatch on either side of 2^19 and 2^22, a pool smaller than the
dispatch), the same bits in every run, and work that follows on another stream
waits for the dispatch."""
import numpy as np
import pytest

from stargaze_b200 import workloads as W
from stargaze_b200.pathtracer import PathTracer
from test_wavefront import assert_same_image, render, small_terrain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp,pool", [
    (1, 1, 1, 0), (16, 16, 1, 0), (17, 15, 3, 0),
    (512, 512, 2, 0), (512, 513, 2, 0),      # 2^19 samples of whole tiles, and one row of tiles more
    (1024, 1024, 4, 0), (1024, 1025, 4, 0),  # 2^22
    (256, 256, 4, 65536),                    # two iterations take the samples
])
@pytest.mark.parametrize("scene", ["rings", "terrain"])
def test_every_rule_renders_the_megakernel_image(scene, width, height, spp, pool):
    wl = W.rings_1080p(width, height) if scene == "rings" else small_terrain(width, height)
    mega, _, _ = render(wl, "megakernel", 2, spp)
    wave, _, n = render(wl, "wavefront", 2, spp, pool=pool)
    again, _, _ = render(wl, "wavefront", 2, spp, pool=pool)
    assert n == 2 * spp
    assert np.array_equal(wave, again)
    if width > 17:
        assert_same_image(wave, mega)


def test_reading_on_another_stream_waits_for_the_dispatch():
    import torch

    wl = W.rings_1080p(640, 360)
    images = []
    for side in (None, torch.cuda.Stream()):
        t = PathTracer((wl.width, wl.height), W.render_options(wl, 16, noise_seed=3))
        W.upload_workload(t, wl)
        for _ in range(3):
            t.encode(wl.frame, side)
        images.append(t.read_pixels())
        t.close()
    assert np.array_equal(images[0], images[1])
