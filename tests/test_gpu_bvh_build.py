"""The locator's BVH-order build against the oracle's sequential one, through what it decides:
located faces, hit counts and positions of query points, bit for bit. Sizes around the 1024
faces below which a subtree is finished in one block (one block, a partly filled second
window, several levels of large nodes), and meshes that drive the partition's special cases:
centroids on split values, many equal centroids, one face split off per level down to the depth
limit, strongly unequal subtrees."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n, kind):
    from otmap_b200 import otmap as ot

    xy = ot.grid_vertices(n)
    rng = np.random.default_rng(n)
    if kind == "snapped":
        xy = np.round((xy + rng.uniform(-0.4, 0.4, xy.shape) / n) * 16) / 16
    elif kind == "warped":
        xy = np.stack([xy[:, 0] ** 9, 1 - (1 - xy[:, 1]) ** 5], axis=1)
    elif kind == "flat":
        xy[:, 1] = 0.5
    elif kind == "point":
        inner = rng.uniform(size=xy.shape[0]) < 0.97
        xy[inner] = 0.5
    return np.ascontiguousarray(xy)


@pytest.mark.parametrize("kind", ["grid", "snapped", "warped", "flat", "point"])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 45, 46, 64, 100, 151])
def test_inversion_matches_oracle(oracle_port, n, kind):
    from otmap_b200 import otmap as ot

    xy = _mesh(n, kind)
    rng = np.random.default_rng(5)
    density = rng.uniform(0.5, 2.0, n * n)
    pick = rng.choice(xy.shape[0], size=min(xy.shape[0], 120), replace=False)
    pts = np.concatenate([np.clip(xy[pick], 0, 1), 0.5 * (xy[pick] + xy[np.roll(pick, 1)]).clip(0, 1),
                          rng.uniform(size=(150, 2))])
    q, faces, hits, _ = oracle_port.apply_inverse(xy, density, n, pts)
    m = ot.TransportMap(n, xy, density)
    p = np.ascontiguousarray(pts.copy())
    face = np.empty(len(p), dtype=np.int32)
    nh = np.empty(len(p), dtype=np.int32)
    m.apply_inverse(p, face, nh)
    m.release()
    assert np.array_equal(nh, hits)
    few = hits <= 8  # the hits kept in order per point
    assert np.array_equal(face[few], faces[few])
    assert np.array_equal(p[few], q[few], equal_nan=True)
