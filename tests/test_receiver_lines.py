"""Receiver grids whose rows run along x, y or z (the axis with most cells), and
launches whose reception spheres are far wider than a cell: lines and thin
slabs of receivers on the small scene against the oracle, on the fast capture
path and on the one that counts stages."""
import numpy as np
import pytest

import oracle as orc
from helpers import field_close, path_keys
from sbrsolver_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [2, 4])
@pytest.mark.parametrize("axis,thick", [(0, 0.0), (1, 0.0), (2, 0.0), (1, 3.0), (2, 3.0)])
def test_receivers_along_each_axis(built, axis, thick, level):
    wl = scenes.small_scene()
    n = 301
    rng = np.random.default_rng(axis)
    rx = np.array([3.0, -4.0, 1.5]) + rng.uniform(0, 1, (n, 3)) * thick
    rx[:, axis] = np.linspace(1.0, 90.0, n)
    q = wl.request
    q.rx, q.tessellation, q.max_reflection, q.max_transmission = rx, level, 2, 1
    ref = orc.solve(orc.OracleScene.from_scene(wl.scene), q, wl.scene.materials)
    sc = api.DeviceScene.from_scene(wl.scene)
    for stage in (False, True):
        res = api.solve(sc, api.request_from_workload(q, stage_counts=stage))
        assert path_keys(res.paths) == path_keys(ref["paths"])
        assert res.counts["corrected"] == ref["counts"]["corrected"]
        if stage:
            assert res.counts["captured"] == ref["counts"]["captured"]
        assert not field_close(res.field, ref["field"])
    sc.close()
