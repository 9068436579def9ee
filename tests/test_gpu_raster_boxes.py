"""The rasterizer's paths by size of a face's pixel box, bit-exact against the oracle: boxes at
and around the 32 pixels that a warp tests in common, large ones spread over warps by chunks of
128 pixels, empty ones (faces off the image or beyond its edge), and folded faces whose
bilinear solve fails (decided by the sequential loop's stale weights), fewer and more of
them than the list of such tests holds."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n, kind, seed):
    from otmap_b200 import otmap as ot

    xy = ot.grid_vertices(n)
    rng = np.random.default_rng(seed)
    if kind == "smooth":
        x, y = xy[:, 0].copy(), xy[:, 1].copy()
        xy[:, 0] += 0.06 * np.sin(2 * np.pi * x) * np.cos(np.pi * y)
        xy[:, 1] += 0.06 * np.sin(2 * np.pi * y) * np.cos(np.pi * x)
    elif kind == "folded":
        xy += rng.uniform(-0.9, 0.9, xy.shape) / n
    elif kind == "shifted":
        xy = xy * 1.3 - 0.17
    return np.ascontiguousarray(xy)


@pytest.mark.parametrize("n,rows,cols", [(1, 33, 65), (2, 11, 200), (16, 80, 96), (16, 81, 64), (40, 40, 40),
                                         (61, 300, 347), (100, 64, 1)])
@pytest.mark.parametrize("kind", ["smooth", "folded", "shifted"])
def test_raster_matches_oracle(oracle_port, n, rows, cols, kind):
    from otmap_b200 import otmap as ot

    xy = _mesh(n, kind, 7 * n + rows)
    density = np.random.default_rng(n).uniform(0.5, 2.0, n * n)
    img = np.empty((rows, cols))
    ot.rasterize_image(xy, density, img, n=n)
    assert np.array_equal(img, oracle_port.rasterize(xy, n, density, rows, cols))
