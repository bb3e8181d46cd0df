"""Search BVH levels whose segments differ in length: a detailed object among
spread triangles, and thousands of triangles with one centroid (median splits).
The blocks are wide enough for the longest segment, and the device's tree is the
host's."""
import os
import subprocess

import numpy as np
import pytest

from sbrsolver_gb300 import api, build, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_long_segment_gets_more_than_a_warp(tmp_path):
    exe = str(tmp_path / "segment_threads_check")
    build.run([build._nvcc(), *build.ARCH, "-std=c++17",
               "-I", os.path.join(ROOT, "sbrsolver_gb300", "csrc"),
               os.path.join(ROOT, "tests", "cpp", "segment_threads_check.cu"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["object", "one centroid"])
def test_uneven_segments_give_the_hosts_tree(built, kind):
    rng = np.random.default_rng(9)
    c = rng.uniform(-500, 500, (20000, 1, 3)) * np.array([1, 1, 0.1])
    tri = [c + rng.normal(0, 0.6, (20000, 3, 3))]
    if kind == "object":
        c = rng.uniform(-1, 1, (8000, 1, 3)) + np.array([37.0, 21.0, 3.0])
        tri.append(c + rng.normal(0, 0.01, (8000, 3, 3)))
    else:  # boxes symmetric about one point, in FP32 too
        half = rng.integers(1, 1024, (3000, 1, 3)) / 1024.0
        at = np.array([37.0, 21.0, 3.0])
        third = rng.integers(-1023, 1024, (3000, 1, 3)) / 1024.0 * half
        tri.append(np.concatenate([at - half, at + half, at + third], 1))
    tri = np.concatenate(tri).astype(np.float32)
    e1, e2 = (tri[:, k].astype(np.float64) - tri[:, 0] for k in (1, 2))
    n = np.cross(e1, e2)
    ok = np.linalg.norm(n, axis=1) > 0
    tri, n = tri[ok], n[ok]
    nrm = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)
    mesh = api.Mesh(tri, nrm, np.zeros(len(tri), np.int32))
    mats = [api.MaterialProperties(*m) for m in scenes.small_scene().scene.materials]
    dev, host = (api.DeviceScene(mesh, mats, host_prep=h) for h in (False, True))
    a, b = dev.search_bvh(), host.search_bvh()
    assert a["max_depth"] == b["max_depth"]
    np.testing.assert_array_equal(a["order"], b["order"])
    np.testing.assert_array_equal(a["nodes"], b["nodes"])
    dev.close()
    host.close()
