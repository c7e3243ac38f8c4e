"""Camera rays skip the bodies and rings their 16x16 tile cannot meet, and tiles
that can meet nothing are not traced. The same scene padded past 32 bodies with
spheres of radius zero, which no ray meets, is traced without either: the images
are equal bit for bit. Seeded scenes: bodies and rings at every orientation and
size, an observer on the ground, close to a ring's plane, inside a ring's radius,
narrow and wide fields, images whose sides are no multiples of the tile."""
import numpy as np
import pytest

from stargaze_b200 import workloads as W
from stargaze_b200.pathtracer import PathTracer
from stargaze_b200.scene import body, frame, ringed

pytestmark = pytest.mark.gpu

SIZES = [(129, 70), (64, 48), (33, 97), (200, 112)]


def unit(v):
    return v / np.linalg.norm(v)


def scene(seed, width, height):
    rng = np.random.default_rng(seed)
    f = frame()
    f.globals.viewport[:] = [float(width), float(height), 1.0, width / height]
    f.globals.cam_forward[3] = float(10.0 ** rng.uniform(-2.0, 0.3))
    tangent = f.globals.cam_forward[3]
    f.bodies = [body(unit(rng.normal(size=3)) * 400.0, 4.0, [4000.0] * 3, True)]
    for k in range(3):  # in view, from points to most of the frame
        depth = rng.uniform(3.0, 40.0)
        c = [rng.uniform(-1.2, 1.2) * tangent * depth * width / height, rng.uniform(-1.2, 1.2) * tangent * depth, -depth]
        radius = depth * tangent * 10.0 ** rng.uniform(-2.0, -0.3)
        b = ringed(c, radius, unit(rng.normal(size=3)), rng.uniform(0.2, 2.0)) if k else body(c, radius, [0.5] * 3, False)
        b.color[:] = [0.6, 0.5, 0.4]
        f.bodies.append(b)
    if seed % 2:  # the ground under the observer, two metres in a planet's radius
        down = unit(rng.normal(size=3))
        radius = 4.0e-5
        f.bodies.append(body(down * radius * (1.0 + 10.0 ** rng.uniform(-6.3, -2.0)), radius, [0.4] * 3, False))
    if seed % 3 == 0:  # a ring around the observer, its plane close by
        pole = unit(rng.normal(size=3))
        side = unit(np.cross(pole, rng.normal(size=3)))
        f.bodies.append(ringed(side * 1.7 + pole * rng.uniform(-0.05, 0.05), 1.0, pole, 0.8))
    return f


def render(f, width, height, seed):
    wl = W.Workload("tiles", f, width, height, 6, 4, {}, "")
    t = PathTracer((width, height), W.render_options(wl, 6, noise_seed=seed))
    t.encode(f)
    image = t.read_pixels()
    t.close()
    return image


@pytest.mark.parametrize("seed", range(24))
def test_culled_image_equals_unculled(seed):
    width, height = SIZES[seed % len(SIZES)]
    f = scene(seed, width, height)
    culled = render(f, width, height, seed)
    padded = f.copy()
    padded.bodies += [body([0.0, 0.0, 5.0 + k], 0.0, [0.0] * 3, False) for k in range(33 - len(f.bodies))]
    full = render(padded, width, height, seed)
    assert np.isfinite(full).all()
    assert np.array_equal(culled, full)
