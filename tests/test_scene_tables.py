"""Scene tables formed on the device from the host's records, which pass through
a buffer of 65,536 triangles: scenes that fill it exactly, by one triangle less
or more, against the oracle, also after the mesh order is set
anew."""
import numpy as np
import pytest

import oracle as orc
from helpers import field_close, path_keys
from sbrsolver_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 65536, 65537])
def test_tables_across_the_buffer(built, n):
    wl = scenes.small_scene()
    rng = np.random.default_rng(n)
    c = rng.uniform(-60, 60, (n, 1, 3)) * np.array([1, 1, 0.2]) + np.array([0, 0, 12.0])
    tri = (c + rng.normal(0, 0.6, (n, 3, 3))).astype(np.float32)
    e1, e2 = (tri[:, k].astype(np.float64) - tri[:, 0] for k in (1, 2))
    nrm = np.cross(e1, e2)
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    q = wl.request
    q.tx = np.array([0.0, 0.0, 12.0])
    q.rx = np.array([0.0, 0.0, 12.0]) + rng.uniform(-8, 8, (200, 3))
    q.tessellation, q.max_reflection, q.max_transmission = 4, 2, 1
    mat = rng.integers(0, len(wl.scene.materials), n).astype(np.int32)
    scene = scenes.Scene("random", tri, nrm, mat, wl.scene.materials)
    ref = orc.solve(orc.OracleScene.from_scene(scene), q, scene.materials)
    sc = api.DeviceScene.from_scene(scene)
    req = api.request_from_workload(q)
    a = api.solve(sc, req)
    assert a.counts["segments"] == ref["counts"]["segments"]
    assert path_keys(a.paths) == path_keys(ref["paths"])
    assert not field_close(a.field, ref["field"])
    sc.set_mesh_order(sc.mesh_order())
    b = api.solve(sc, req)
    assert np.array_equal(a.field, b.field)
    sc.close()
