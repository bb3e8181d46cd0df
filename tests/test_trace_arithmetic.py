"""What the trace stage decides without the reference's FP64 instructions: FP64
operations in integer arithmetic (csrc/sbr_soft64.cuh), the FP32 triangle
filter's margin (tri_classify), and the one-box reachability check
(leaf_reachable in csrc/sbr_kernels.cuh), each against plain FP64."""
import os
import subprocess

import numpy as np
import pytest

import oracle as orc
from helpers import field_close, path_keys
from sbrsolver_gb300 import api, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
F = np.float32
EPS = F(1.1920928955078125e-07)


@pytest.mark.parametrize("seed_error", ["0.0f", "2.3e-7f", "-2.3e-7f"])
def test_soft64_gives_the_hosts_bits(tmp_path, seed_error):
    exe = str(tmp_path / "soft64_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off",
                    f"-DSBR_SOFT64_SEED_ERROR={seed_error}",
                    "-I", os.path.join(ROOT, "sbrsolver_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "soft64_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _cross(a, b):
    return np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                     a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)


def _dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def test_triangle_filter_margin():
    """tri_classify's FP32 arithmetic with its 2^-18 margin on rays aimed at a
    triangle's edges (within a few margins), from 0.1 m to 3 km away: a ray it
    drops misses in FP64, and one whose u and v it calls sure passes FP64's
    tests of them."""
    rng = np.random.default_rng(3)
    n, K = 400000, F(2.0 ** -18)
    size = 10 ** rng.uniform(-1, 2.5, (n, 1))
    c0 = rng.uniform(-1000, 1000, (n, 3))
    v = [(c0 + rng.normal(0, 1, (n, 3)) * size).astype(F).astype(np.float64) for _ in range(3)]
    e1, e2 = v[1] - v[0], v[2] - v[0]
    # a point near an edge or corner, in barycentric coordinates
    a = rng.uniform(0, 1, (n, 1))
    j = rng.normal(0, 1, (n, 2)) * 10 ** rng.uniform(-8, -2, (n, 1))
    edge = rng.integers(0, 3, (n, 1))
    b1 = np.where(edge == 0, 0.0, a) + j[:, :1]
    b2 = np.where(edge == 0, a, np.where(edge == 1, 0.0, 1.0 - a)) + j[:, 1:]
    p = v[0] + b1 * e1 + b2 * e2
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = p - d * 10 ** rng.uniform(-1, 3.5, (n, 1))
    # FP64, the reference's order
    h = _cross(d, e2)
    det = _dot(e1, h)
    with np.errstate(all="ignore"):
        f = 1.0 / det
        s = o - v[0]
        u, q = f * _dot(s, h), _cross(s, e1)
        w, t = f * _dot(d, q), f * _dot(e2, q)
        par = (det > -float(EPS)) & (det < float(EPS))
        uv = ~((u < 0) | (u > 1) | (w < 0) | (u + w > 1))
        hit = ~par & uv & (t > float(EPS))
    # FP32
    D, O, V, E1, E2 = (x.astype(F) for x in (d, o, v[0], e1, e2))
    H, S = _cross(D, E2), O - V
    A, U, Q = _dot(E1, H), _dot(S, H), _cross(S, E1)
    Vv, W = _dot(D, Q), _dot(E2, Q)
    norm = lambda x: np.sqrt(_dot(x, x))  # noqa: E731
    up = F(1.0001)
    ne1, ne2, nd, ns = norm(E1) * up, norm(E2) * up, norm(D), norm(O) + norm(V) * up
    ea, eU, eV, eW = K * ne1 * ne2 * nd, K * ns * nd * ne2, K * ns * ne1 * nd, K * ns * ne1 * ne2
    m = np.abs(A)
    near = m <= EPS + ea
    sg = np.where(A < 0, F(-1), F(1))
    U, Vv, W = U * sg, Vv * sg, W * sg
    with np.errstate(all="ignore"):
        thi = (W + eW) / (m - ea)
    drop = ~near & ((U < -eU) | (Vv < -eV) | (U > m + ea + eU) | (U + Vv > m + ea + eU + eV) |
                    (thi <= EPS * F(0.5)))
    sure = ~near & ~drop & (U > eU) & (Vv > eV) & (U + Vv < m - ea - eU - eV)
    assert not (drop & hit).any()
    assert (uv | par)[sure].all()
    assert min(hit.sum(), sure.sum(), drop.sum()) > 10000  # every decision occurs


def _slab64(bb, o, d):
    """The reference's slab test (BVHNode.h:64-85), its NaN rules included."""
    n = len(o)
    tmax, tmin, ok = np.full(n, np.inf), np.full(n, -np.inf), np.ones(n, bool)
    with np.errstate(all="ignore"):
        for i in range(3):
            t1, t2 = (bb[:, i] - o[:, i]) / d[:, i], (bb[:, 3 + i] - o[:, i]) / d[:, i]
            tn, tf = np.where(t2 < t1, t2, t1), np.where(t1 < t2, t2, t1)
            tmax, tmin = np.where(tf < tmax, tf, tmax), np.where(tmin < tn, tn, tmin)
            ok &= ~(tmin > tmax)
    return ok


@pytest.mark.parametrize("zero_axes", [(), (0,), (1, 2)])
def test_leaf_box_decides_for_its_ancestors(zero_axes):
    """Random nested boxes (shared planes, flat ones, signed zeros) and rays
    through or past the inner one's corners: where it passes the reference's
    slab test, so do the outer ones, provided a zero direction component's
    planes lie strictly on either side of the origin; both cases occur."""
    rng = np.random.default_rng(5)
    n = 200000
    lo = rng.integers(-8, 8, (n, 3)).astype(np.float64)
    hi = lo + rng.integers(0, 4, (n, 3))
    grow = rng.integers(0, 3, (n, 6))
    outer = np.concatenate([lo - grow[:, :3], hi + grow[:, 3:]], 1)
    inner = np.concatenate([np.where((lo == 0) & (rng.random((n, 3)) < 0.5), -0.0, lo), hi], 1)
    o = rng.uniform(-12, 12, (n, 3))
    snap = rng.random((n, 3)) < 0.3
    o = np.where(snap, np.where(rng.random((n, 3)) < 0.5, lo, hi), o)
    target = np.where(rng.random((n, 3)) < 0.7, np.where(rng.random((n, 3)) < 0.5, lo, hi),
                      rng.uniform(lo, np.maximum(hi, lo + 1e-9)))
    d = (target - o) * 10 ** rng.uniform(-3, 3, (n, 1))
    d = np.where(d == 0, 1e-3, d)
    ok = np.ones(n, bool)
    for a in zero_axes:
        d[:, a] = np.where(rng.random(n) < 0.5, 0.0, -0.0)
        o[:, a] = np.where(rng.random(n) < 0.5, rng.uniform(lo[:, a] - 0.5, hi[:, a] + 0.5), o[:, a])
        ok &= (o[:, a] > lo[:, a]) & (o[:, a] < hi[:, a])
    leaf = _slab64(inner, o, d) & ok
    assert leaf.sum() > 1000
    assert _slab64(outer, o, d)[leaf].all()


@pytest.mark.gpu
@pytest.mark.parametrize("tx", [(0.0, 0.0, 20.0),        # many rays with a zero component
                                "wall",                  # ... sliding along a wall's plane
                                (1e-40, 0.0, 20.0)])     # outside the integer arithmetic's range
def test_axis_parallel_rays_match_the_oracle(built, tx):
    wl = scenes.urban_scene(level=4, rx_pitch=50.0, max_reflection=3, max_transmission=1)
    if tx == "wall":  # the plane of the first building's first side wall
        w = wl.scene.tri[2 + 8:, :, 0]
        tx = (float(w[0, 0]), float(wl.scene.tri[2:14, :, 1].min()) - 7.0, 5.0)
    wl.request.tx = tx
    ref = orc.solve(orc.OracleScene.from_scene(wl.scene), wl.request, wl.scene.materials)
    sc = api.DeviceScene.from_scene(wl.scene)
    res = api.solve(sc, api.request_from_workload(wl.request))
    assert res.counts["segments"] == ref["counts"]["segments"]
    assert path_keys(res.paths) == path_keys(ref["paths"])
    for p, q in zip(res.paths, ref["paths"]):
        np.testing.assert_array_equal(p["points"], q["points"])
    assert not field_close(res.field, ref["field"])
    sc.close()
