"""The result the device writes into host staging: paths in receiver order with
their rays packed, at no receivers, no paths, one, and more than the first
staging holds (it is then grown and written again), with the FP64 shadow field
and over several requests."""
import numpy as np
import pytest

from sbrsolver_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("counts", [[0], [1], [33, 0, 4], [2500, 700]])
def test_result_is_packed_in_receiver_order(built, counts, precision):
    wl = scenes.small_scene()
    q = wl.request
    rng = np.random.default_rng(len(counts))
    req = []
    for n in counts:
        q.rx = np.array([1.0, -8.0, 1.5]) + rng.uniform(0, 1, (n, 3)) * np.array([60.0, 16.0, 3.0])
        q.tessellation, q.max_reflection, q.max_transmission = 3, 2, 1
        req.append(api.request_from_workload(q, precision=precision, field_check=True))
    sc = api.DeviceScene.from_scene(wl.scene)
    a = api.solve(sc, req, with_paths="arrays")
    b = api.solve(sc, req, with_paths="arrays")  # staging is large enough now
    sc.close()
    assert a.field.shape == (sum(counts), 3) and np.array_equal(a.field, b.field)
    if not a.counts["paths"]:
        assert not a.paths and not a.field.any()
        return
    p = a.paths
    for k in p:
        assert np.array_equal(p[k], b.paths[k]), k
    assert np.array_equal(p["ray_offset"], np.cumsum(p["n_rays"]) - p["n_rays"])
    assert p["n_rays"].sum() == len(p["tri"]) == len(p["points"]) == a.counts["rays"]
    order = np.lexsort((p["heap"], p["launch"], p["receiver"], p["request"]))
    assert np.array_equal(order, np.arange(len(order)))
    # a path runs from its transmitter through its points to its receiver
    first = np.cumsum([0] + counts)
    rx = np.concatenate([np.asarray(r[1]).reshape(-1, 3) for r in req])
    for i in range(len(order)):
        o, n = p["ray_offset"][i], p["n_rays"][i]
        pts = p["points"][o:o + n].reshape(n, 2, 3)
        assert np.array_equal(pts[0, 0], np.asarray(q.tx, np.float64))
        assert np.array_equal(pts[1:, 0], pts[:-1, 1])
        assert np.array_equal(pts[-1, 1], rx[first[p["request"][i]] + p["receiver"][i]])
    if precision == "fp64":  # the field is the ordered sum of the paths' fields
        f = np.zeros((sum(counts), 6))
        for i in range(len(order)):
            f[first[p["request"][i]] + p["receiver"][i]] += p["field"][i]
        assert np.array_equal(f.view(np.complex128).reshape(-1, 3), a.field)
