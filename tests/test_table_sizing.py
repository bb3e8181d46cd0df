"""Tables sized by the solve's own size class: solves of very different sizes in
turn on one workspace give what each gives alone, and replay as graphs."""
import numpy as np
import pytest

from helpers import path_keys
from sbrsolver_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [(1, 7), (7, 1), (5, 6)])
def test_sizes_in_turn(built, levels):
    wl = scenes.small_scene()
    q = wl.request
    rng = np.random.default_rng(7)
    req = []
    for level in levels:
        q.tessellation, q.max_reflection, q.max_transmission = level, 2, 1
        n = 3000 if level < 5 else 40
        q.rx = np.array([1.0, -8.0, 1.5]) + rng.uniform(0, 1, (n, 3)) * np.array([60.0, 16.0, 3.0])
        req.append(api.request_from_workload(q))
    sc = api.DeviceScene.from_scene(wl.scene)
    alone = [api.solve(sc, r) for r in req]
    for turn in range(4):
        for r, want in zip(req, alone):
            got = api.solve(sc, r)
            assert path_keys(got.paths) == path_keys(want.paths)
            assert np.array_equal(got.field, want.field)
            assert got.counts["segments"] == want.counts["segments"]
            if turn == 3:
                assert got.counts["pipeline_graph"] == 1
    sc.close()
