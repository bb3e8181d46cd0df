"""The device reference BVH's partition rounds on segments just above the longest
a block sorts by itself, and at the edges of the rounds' tiles, with long runs
of equal keys: same tree and order as the host build."""
import numpy as np
import pytest

from sbrsolver_gb300 import api, scenes
from test_gpu_scene_prep import _tie_heavy_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048, 2049, 3071, 3072, 3073, 4097, 9217])
def test_rounds_at_tile_edges(built, n):
    tri, nrm = _tie_heavy_scene(n, n)
    mats = [api.MaterialProperties(*m) for m in scenes.small_scene().scene.materials]
    mesh = api.Mesh(tri, nrm, np.zeros(n, np.int32))
    a = api.DeviceScene(mesh, mats)
    b = api.DeviceScene(mesh, mats, host_prep=True)
    ra, rb = a.reference_bvh(), b.reference_bvh()
    for key in ("links", "order"):
        np.testing.assert_array_equal(ra[key], rb[key])
    np.testing.assert_array_equal(a.mesh_order(), b.mesh_order())
    a.close()
    b.close()
