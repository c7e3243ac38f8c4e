"""The terrain walk over its node and leaf records against the oracle's
traversal (separate child boxes, general triangle test): distances bit for
bit, normals within the 2e-6 of the other landscape tests. Grids from the
single leaf (2 cells) over the largest one with three-float normals (1024)
to a compact one (2048); rays with zero direction components, origins on grid
lines and vertices, rays from below and beyond the edge."""
import numpy as np
import pytest

import known_answers as ka
from stargaze_b200 import PathTracer
from stargaze_b200 import terrain as T

pytestmark = pytest.mark.gpu


def rays(cells, heights, seed):
    rng = np.random.default_rng(seed)
    n = 384
    c = T.coordinates(cells)
    o = np.stack([rng.uniform(-17000, 17000, n), rng.uniform(-50, 500, n), rng.uniform(-17000, 17000, n)], axis=1)
    d = rng.normal(size=(n, 3)) * [1.0, 0.4, 1.0]
    # Origins on grid columns, rows and vertices.
    on = rng.integers(0, cells + 1, (n, 2))
    o[0::4, 0] = c[on[0::4, 0]]
    o[1::4, 2] = c[on[1::4, 1]]
    o[2::4, 0], o[2::4, 2] = c[on[2::4, 0]], c[on[2::4, 1]]
    # Directions along and across the axes: one or two exact zeros.
    for k, zero in enumerate(([0], [2], [0, 2], [1], [0, 1])):
        d[5 + k::16, zero] = 0.0
    o[12::16, 1] = -2000.0  # from below
    d[12::16, 1] = np.abs(d[12::16, 1]) + 0.2
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("theme", [0, 3], ids=["forest", "alpine"])
@pytest.mark.parametrize("cells", [2, 4, 128, 1024, 2048])
def test_walk_matches_oracle(cells, theme):
    from oracle.binding import OracleTracer

    heights = T.fbm_heights(cells, seed=cells + theme)
    data = T.pack_terrain(heights, cells)
    o, d = rays(cells, heights, seed=31 * cells + theme)
    results = []
    for tracer in (PathTracer((1, 1), ka.test_options()), OracleTracer((1, 1), ka.test_options())):
        tracer.upload_terrain(data, cells)
        f = ka.terrain_frame(6_371_000.0)
        f.globals.ground_counts[2] = (f.globals.ground_counts[2] & ~255) | theme
        results.append(tracer.terrain_probe(f, o, d))
    cuda, cpu = results
    assert np.array_equal(cuda[:, 3], cpu[:, 3])
    hit = cpu[:, 3] < 1e29
    assert 0.2 < hit.mean() < 0.95
    assert np.abs(cuda[hit, :3] - cpu[hit, :3]).max() < 2e-6
