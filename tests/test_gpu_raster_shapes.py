"""The rasterizer's shapes of launch, bit-exact against the oracle: meshes on both sides of the
face counts at which a warp takes 1, 4, 8 and 32 faces (2368, 9472 and 75776 on 148 SMs), drawn
with boxes below, around and above the 32 and 256 pixels that a warp pools, smooth and folded,
from quads and from triangles."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n, kind):
    from otmap_b200 import otmap as ot

    xy = ot.grid_vertices(n)
    rng = np.random.default_rng(n)
    if kind == "smooth":
        x, y = xy[:, 0].copy(), xy[:, 1].copy()
        xy[:, 0] += 0.06 * np.sin(2 * np.pi * x) * np.cos(np.pi * y)
        xy[:, 1] += 0.06 * np.sin(2 * np.pi * y) * np.cos(np.pi * x)
    else:
        xy += rng.uniform(-0.6, 0.6, xy.shape) / n
    return np.ascontiguousarray(xy)


@pytest.mark.parametrize("n,rows,cols", [(8, 40, 130), (12, 190, 60), (48, 48, 300), (49, 260, 256), (97, 500, 97),
                                         (98, 98, 590), (275, 275, 300), (276, 280, 1200), (20, 330, 320)])
@pytest.mark.parametrize("kind", ["smooth", "folded"])
def test_quads(oracle_port, n, rows, cols, kind):
    from otmap_b200 import otmap as ot

    xy = _mesh(n, kind)
    density = np.random.default_rng(n).uniform(0.5, 2.0, n * n)
    img = np.empty((rows, cols))
    ot.rasterize_image(xy, density, img, n=n)
    assert np.array_equal(img, oracle_port.rasterize(xy, n, density, rows, cols))


@pytest.mark.parametrize("n,rows,cols", [(12, 150, 160), (33, 70, 400), (69, 200, 140)])
def test_triangles_and_quads(oracle_port, n, rows, cols):
    from otmap_b200 import otmap as ot

    xy = _mesh(n, "smooth")
    quads = ot.Mesh.grid(n, xy).face_vertices.reshape(-1, 4)
    faces = []
    for k, q in enumerate(quads):  # every third quad as two triangles
        faces += [q[[0, 1, 2]], q[[0, 2, 3]]] if k % 3 == 0 else [q]
    start = np.cumsum([0] + [len(f) for f in faces]).astype(np.int32)
    mesh = ot.Mesh(xy, start, np.concatenate(faces).astype(np.int32))
    density = np.random.default_rng(n).uniform(0.5, 2.0, len(faces))
    for mode in (ot.RIO_PerFaceDensity, ot.RIO_PerVertexDensity):
        img = np.empty((rows, cols))
        ot.rasterize_image(mesh, density, img, mode)
        want = oracle_port.rasterize_mesh(xy, start, mesh.face_vertices, density, rows, cols,
                                          per_vertex=mode == ot.RIO_PerVertexDensity)
        assert np.array_equal(img, want)
