"""Group markers are skipped by products with the ray's reciprocals where those
are certain, else by the exact divisions: closest hits and visibilities equal
the oracle's (which divides) bit for bit, with rays through the corners and along the
edges and faces of the boxes, axis-parallel ones, and boxes about as far as the
closest hit."""
import numpy as np
import pytest

import known_answers as ka
from stargaze_b200 import PathTracer
from stargaze_b200 import terrain as T
from stargaze_b200.pathtracer import rays_array
from stargaze_b200.scene import AU_M

pytestmark = pytest.mark.gpu


def scene(seed):
    rng = np.random.default_rng(seed)
    f = ka.local_frame(6_371_000.0)
    props = []
    for k in range(40):
        centre = [rng.uniform(-60, 60), rng.uniform(0.5, 12.0), rng.uniform(-60, 60)]
        extent = list(rng.uniform(0.3, 3.0, 3))
        if k % 4 == 0:  # boxes on a lattice share planes with their groups
            centre, extent = [float(v) for v in np.round(centre)], [1.0, 1.0, 1.0]
        kind = [0.0, 1.0, 2.0, 2.25][k % 4]
        props.append(T.primitive(centre, kind, extent, 0.0 if k % 4 != 3 else float(rng.integers(0, 1 << 24)),
                                 (0.3, 0.3, 0.3), 1.0))
    f.ground = T.build_prop_bvh(props, leaf_size=2)
    f.globals.ground_counts[0] = len(f.ground)
    return f, rng


def group_rays(f, rng):
    """Ground-frame origins and directions."""
    origins, targets = [], []
    for p in f.ground:
        if p.center[3] >= 0.0:
            continue
        c, e = np.array(p.center[:3], np.float64), np.array(p.extent[:3], np.float64)
        for sign in rng.choice([-1.0, 0.0, 1.0], (24, 3)):
            origins.append([rng.uniform(-80, 80), rng.uniform(1.0, 30.0), rng.uniform(-80, 80)])
            targets.append(c + sign * e)
        for axis in range(3):  # along a face or an edge, and straight at it
            for _ in range(6):
                t = c + rng.choice([-1.0, 1.0, 0.3], 3) * e
                o = t.copy()
                o[axis] += rng.choice([-1.0, 1.0]) * rng.uniform(5.0, 70.0)
                origins.append(o)
                targets.append(t)
    o, t = np.array(origins), np.array(targets)
    d = t - o
    return o, d / np.linalg.norm(d, axis=1, keepdims=True)


@pytest.mark.parametrize("seed", range(4))
def test_hits_equal_the_oracles(seed):
    from oracle.binding import OracleTracer

    f, rng = scene(seed)
    o, d = group_rays(f, rng)
    g = f.globals
    axes = np.array([g.ground_east[:3], g.ground_up[:3], g.ground_north[:3]], np.float64)
    o = o - [0.0, float(g.ground_east[3]), 0.0]
    rays = rays_array((o @ axes) / AU_M, (d @ axes).astype(np.float32), 0xFFFFFFFF)
    results = [t.closest_hit(f, rays) for t in (PathTracer((1, 1), ka.test_options()),
                                                OracleTracer((1, 1), ka.test_options()))]
    cuda, cpu = results
    assert np.array_equal(cuda["index"], cpu["index"])
    assert np.array_equal(cuda["distance"], cpu["distance"])
    assert ((cpu["index"] > 0x80000000) & (cpu["index"] < 0x80100000)).mean() > 0.1
