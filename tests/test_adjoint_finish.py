"""When the rest of a staged replay goes to the finish kernel: after the first
iteration up to 2^16 samples, else on a landscape once the GPU finds few paths
left, in celestial frames once the host has seen that. On either side of the
lines, and with a pool so small that a second batch needs the slots that the first
one's finish kernel kept, the gradients are the per-pixel kernel's."""
import numpy as np
import pytest

from stargaze_b200 import workloads as W
from test_wave_adjoint import assert_same_gradient, both_adjoints

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp,pool", [
    (128, 128, 4, 0), (128, 129, 4, 0),  # 2^16 samples of whole tiles, and one row of tiles more
    (128, 128, 4, 16384),                # 2^16, of which the pool holds a quarter
    (256, 256, 8, 0),                    # 2^19: more than 2^17 paths at first
    (64, 48, 128, 2048),                 # two batches of 64 samples
])
def test_celestial_gradients(width, height, spp, pool):
    wl = W.rings_1080p(width, height, spp)
    staged, ref = both_adjoints(wl, spp, seed=21, pool=pool)
    assert staged.dropped == 0 and ref.dropped == 0
    assert_same_gradient(staged.ring_tau[0, :512], ref.ring_tau[0, :512], "ring_tau")
    assert_same_gradient(staged.ring_albedo, ref.ring_albedo, "ring_albedo")
    assert_same_gradient(staged.body_color, ref.body_color, "body_color")


@pytest.mark.parametrize("width,height,spp,pool", [(128, 129, 4, 0), (64, 48, 128, 2048)])
def test_landscape_gradients(width, height, spp, pool):
    wl, land = W.terrain_1080p(width, height, spp, cells=256, rocks=60, foliage=60)
    land.albedo_map = np.random.default_rng(4).uniform(0.05, 0.6, (64, 64)).astype(np.float32)
    land.map_extent = 2000.0
    staged, ref = both_adjoints(wl, spp, seed=22, land=land, pool=pool)
    assert staged.dropped == 0 and ref.dropped == 0
    assert_same_gradient(staged.albedo_map, ref.albedo_map, "albedo_map")
    assert_same_gradient(staged.body_color, ref.body_color, "body_color")
