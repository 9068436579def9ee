"""The BVH-order build where its two phases meet: a node of at most 512 faces is set aside and
finished in one block. 22^2 = 484 faces are set aside at the root, 23^2 = 529 are split once or
more over the whole array first; the meshes and the comparison are those of the build's other
sizes."""

import pytest
import test_gpu_bvh_build as build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["grid", "snapped", "warped", "flat", "point"])
@pytest.mark.parametrize("n", [4, 10, 16, 21, 22, 23, 24, 30])
def test_root_set_aside_and_split(oracle_port, n, kind):
    build.test_inversion_matches_oracle(oracle_port, n, kind)
