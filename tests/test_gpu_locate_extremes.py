"""The point locator on meshes far from any map: faces that each cover a third of the square (their
lists over n^2 bins would be longer than an int can index: fewer bins are taken), against the
oracle; and a mesh with vertices that are not numbers, whose other faces are located as without them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inverse(n, xy, density, pts):
    from otmap_b200 import otmap as ot

    m = ot.TransportMap(n, xy, density)
    p = np.ascontiguousarray(pts.copy())
    face, hits = np.empty(len(p), dtype=np.int32), np.empty(len(p), dtype=np.int32)
    missing = m.apply_inverse(p, face, hits)
    m.release()
    return p, face, hits, missing


@pytest.mark.parametrize("n", [40, 288])  # 288: 82944 faces of 0.36 * 82944 bins, 2.5e9 entries
def test_random_vertices(oracle_port, n):
    rng = np.random.default_rng(n)
    xy = np.ascontiguousarray(rng.uniform(size=((n + 1) ** 2, 2)))
    density = rng.uniform(0.5, 2.0, n * n)
    pts = np.concatenate([rng.uniform(size=(30, 2)), rng.uniform(0.0, 0.004, size=(20, 2))])
    q, faces, hits, _ = oracle_port.apply_inverse(xy, density, n, pts)
    p, face, nh, _ = _inverse(n, xy, density, pts)
    assert np.array_equal(nh, hits)
    few = hits <= 8  # the hits kept in order per point
    assert np.array_equal(face[few], faces[few])
    assert np.array_equal(p[few], q[few], equal_nan=True)


def test_vertices_that_are_not_numbers():
    from otmap_b200 import otmap as ot

    n = 40
    clean = ot.grid_vertices(n)
    rng = np.random.default_rng(1)
    clean += rng.uniform(-0.2, 0.2, clean.shape) / n
    bad = clean.copy()
    for v in (5, 900, 901, 942, 1680):
        bad[v] = np.nan
    bad[300, 0] = np.nan
    density = rng.uniform(0.5, 2.0, n * n)
    pts = rng.uniform(0.02, 0.98, size=(3000, 2))
    want, face, hits, _ = _inverse(n, clean, density, pts)
    got, face_b, hits_b, missing = _inverse(n, bad, density, pts)
    i, j = face // n, face % n
    corners = np.stack([(i + a) * (n + 1) + j + b for a in (0, 1) for b in (0, 1)])
    whole = (hits == 1) & ~np.isnan(bad[corners]).any(axis=(0, 2))
    assert whole.sum() > 2900
    assert np.array_equal(face_b[whole], face[whole]) and np.array_equal(got[whole], want[whole])
    assert missing <= (~whole).sum()
