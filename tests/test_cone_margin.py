"""The correction cone's margin, 2 m with m = 2^-21 |n| (cmax + |img| + |T| + 1)
(sbr_capture.cuh, planes formed in FP64 by k_class_cones): the FP32 test of a
receiver, and of the grid cell around it, never rejects a point of the exact
cone, also for triangles seen at a grazing angle or from far away, where the
cone is thinner than the margin."""
import numpy as np

F = np.float32
K = F(2.0 ** -21)


def test_cone_margin_keeps_every_point_of_the_cone():
    rng = np.random.default_rng(12)
    n, cmax = 300000, 1500.0
    size = 10 ** rng.uniform(-0.5, 2, (n, 1))
    c0 = rng.uniform(-1000, 1000, (n, 3))
    v = [(c0 + rng.normal(0, 1, (n, 3)) * size).astype(F).astype(np.float64) for _ in range(3)]
    img = v[0] + rng.normal(0, 1, (n, 3)) * 10 ** rng.uniform(0, 3.5, (n, 1))
    # half of the image sources close to the triangle's plane (grazing)
    nt = np.cross(v[1] - v[0], v[2] - v[0])
    nt /= np.linalg.norm(nt, axis=1, keepdims=True)
    h = ((img - v[0]) * nt).sum(1, keepdims=True)
    img -= np.where(rng.random((n, 1)) < 0.5, h * (1 - 10 ** rng.uniform(-4, -1, (n, 1))), 0.0) * nt
    g = (v[0] + v[1] + v[2]) / 3.0
    norm = lambda x: np.linalg.norm(x, axis=1)  # noqa: E731
    tmag = norm(img) + norm(v[0]) + norm(v[1] - v[0]) + norm(v[2] - v[0]) + 1.0
    # a receiver on the line through a point of an edge (or the inside), jittered
    k = rng.integers(0, 3, n)
    e0 = np.choose(k[:, None], v)
    e1 = np.choose((k[:, None] + 1) % 3, v)
    p = e0 + rng.uniform(0, 1, (n, 1)) * (e1 - e0)
    p += (g - p) * 10 ** rng.uniform(-14, 0, (n, 1))
    x = img + rng.uniform(1.0, 3.0, (n, 1)) * (p - img)
    x = x.astype(F)  # the grid holds receivers rounded to FP32
    inside, passes, usable = (np.ones(n, bool) for _ in range(3))
    x64 = x.astype(np.float64)
    for j in range(3):
        a, b = v[j] - img, v[(j + 1) % 3] - img
        nn = np.cross(a, b)
        gc = (nn * (g - img)).sum(1)
        ln = norm(nn)
        usable &= (ln > 1e-6 * norm(a) * norm(b)) & (np.abs(gc) > 4e-9 * ln * tmag)
        nn *= np.where(gc > 0, 1.0, -1.0)[:, None]
        inside &= (nn * (x64 - img)).sum(1) >= 0
        n32, off = nn.astype(F), (nn * img).sum(1).astype(F)
        m = K * (ln.astype(F) * F(cmax) + (ln * tmag).astype(F))
        lhs = (n32[:, 0] * x[:, 0] + n32[:, 1] * x[:, 1]) + n32[:, 2] * x[:, 2]
        passes &= lhs >= off - F(2) * m
    ok = usable & (norm(x64) <= cmax) & inside
    assert ok.sum() > 20000
    assert passes[ok].all()
