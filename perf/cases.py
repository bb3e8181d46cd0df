"""Performance cases: the calls a user of this framework makes, over the
range of sizes and options in use.

A case is a dict of plain values.  Its "kind" says which public entry points
one pass goes through:

  trace   RTSolver.ExecuteRayTracing, the reference-named call
  solve   api.solve of one request on a resident scene
  batch   api.solve of many transmitters in one call
  serve   api.Server: a burst of mixed requests on two resident scenes
  study   a scene created, solved once and dropped (geometry variants)
  scene   a scene created, its mesh order and coplanar ids read, dropped
  sum     sbr_receiver_field_sum_noalloc on device buffers

Scenes are the repository's own seeded ones (sbrsolver_gb300.scenes): the
ground strip of the reference's main(), the site of ten box buildings, the
urban canyon and the fractal terrain.  A seed moves transmitters and
receivers (and, for study and scene, the geometry); antenna, precision, depth
and size come from the case.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from sbrsolver_gb300 import _lib, api, scenes

# ------------------------------------------------------------------ the cases


def _solve(name, scene, level, r, t, rx, antenna=1, precision="fp64", walls="fresnel",
           size=0, kind="solve"):
    return {"name": name, "kind": kind, "scene": scene, "size": size, "level": level,
            "reflections": r, "transmissions": t, "receivers": rx, "antenna": antenna,
            "precision": precision, "walls": walls}


def listed():
    return [
        # The smallest call: the scene of the reference's main(), two triangles,
        # 162 launch rays and a drive-test line of 3,000 receivers.
        _solve("strip_line", "strip", 2, 1, 0, 3000, kind="trace"),
        # A site check: ten buildings, 40,962 rays, a handful of receivers,
        # half-wave dipole.  Latency and launches count.
        _solve("site_check", "site", 6, 3, 0, 16, antenna=2),
        # One transmitter of a network plan on the urban canyon.
        _solve("canyon_plan", "canyon", 7, 5, 0, 4096, antenna=2, size=400),
        # Indoor penetration: slab walls, two transmissions, a rotated frame,
        # FP32 field with its error bound, an odd number of receivers.
        _solve("canyon_slab", "canyon", 7, 3, 2, 1601, antenna=2, precision="fp32",
               walls="slab", size=400),
        # The headline solve: 2.6M rays, 6 reflections and 1 transmission,
        # 10,000 receivers on a 10 m grid.
        _solve("canyon_full", "canyon", 9, 6, 1, 10000, antenna=0, size=400),
        # Part of a region: 33k triangles, 10 m buildings on terrain, receivers
        # scattered at odd count.
        _solve("terrain_part", "terrain", 8, 4, 1, 7777, antenna=1, size=128),
        # The largest: 580k triangles, 10.5M rays, 8 reflections, 50,000
        # receivers, FP32 field.
        _solve("terrain_full", "terrain", 10, 8, 0, 50000, antenna=2, precision="fp32", size=512),
        # Many transmitters planned in one call, uneven ray budgets and patterns.
        {"name": "canyon_batch", "kind": "batch", "size": 400, "requests": 24, "level_min": 6,
         "level_max": 8, "reflections": 5, "receivers": 4096},
        # A burst of requests at a server holding two scenes.
        {"name": "serve_burst", "kind": "serve", "size": 400, "requests": 20, "level_min": 5,
         "level_max": 8, "receivers_max": 10000, "slots": 2},
        # A design study: a new street layout, one coarse solve of it.
        _solve("street_study", "canyon", 6, 3, 0, 400, antenna=2, size=399, kind="study"),
        # A large terrain model loaded.
        {"name": "terrain_load", "kind": "scene", "scene": "terrain", "size": 512},
        # Path fields summed per receiver inside another framework's pipeline.
        {"name": "field_sum", "kind": "sum", "paths": 120001, "receivers": 20011,
         "precision": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, n):
    return n | 1 if rng.random() < 0.5 else n


def _tree(r, t):
    """Bound on the segments of one launch: interaction sequences with at most
    r reflections and t transmissions."""
    return sum(math.comb(i + j, i) for i in range(r + 1) for j in range(t + 1))


_LARGEST = {"canyon": (10 * 4 ** 9 + 2) * _tree(6, 1), "terrain": (10 * 4 ** 10 + 2) * _tree(8, 0)}


def draw(rng):
    """A case of the same ranges: mostly solves over every scene, depth, level,
    receiver count, antenna and precision, sometimes the other kinds."""
    k = rng.random()
    if k < 0.62:
        scene = rng.choice(["site", "canyon", "canyon", "terrain"])
        t = rng.choice([0, 0, 0, 1, 1, 2])
        r = rng.randint(1, 6 if t else 8)
        size = {"site": 0, "canyon": _log_int(rng, 20, 400), "terrain": rng.choice([64, 128, 256])}[scene]
        top = {"site": 7, "canyon": 9, "terrain": 9}[scene]
        bound = _LARGEST.get(scene, _LARGEST["canyon"]) // 2
        while top > 4 and (10 * 4 ** top + 2) * _tree(r, t) > bound:
            top -= 1
        rx = _odd(rng, _log_int(rng, 16, 512 if scene == "site" else 30000))
        return _solve("", scene, rng.randint(4, top), r, t, rx, antenna=rng.randint(0, 2),
                      precision=rng.choice(["fp64", "fp64", "fp32"]),
                      walls=rng.choice(["fresnel", "fresnel", "slab"]), size=size) | {"name": "drawn"}
    if k < 0.72:
        return {"name": "drawn", "kind": "batch", "size": _log_int(rng, 50, 400),
                "requests": rng.randint(3, 24), "level_min": 5, "level_max": rng.randint(6, 8),
                "reflections": rng.randint(2, 5), "receivers": _odd(rng, _log_int(rng, 256, 4096))}
    if k < 0.78:
        return {"name": "drawn", "kind": "serve", "size": _log_int(rng, 50, 400),
                "requests": rng.randint(4, 20), "level_min": 4, "level_max": rng.randint(6, 8),
                "receivers_max": _log_int(rng, 500, 10000), "slots": rng.randint(1, 3)}
    if k < 0.85:
        return _solve("drawn", "canyon", rng.randint(4, 7), rng.randint(1, 4), 0,
                      _odd(rng, _log_int(rng, 16, 2000)), antenna=rng.randint(0, 2),
                      size=_log_int(rng, 20, 400), kind="study")
    if k < 0.92:
        return {"name": "drawn", "kind": "scene", "scene": rng.choice(["canyon", "terrain"]),
                "size": rng.choice([64, 128, 256])}
    return {"name": "drawn", "kind": "sum", "paths": _odd(rng, _log_int(rng, 1000, 260000)),
            "receivers": _odd(rng, _log_int(rng, 500, 100000)),
            "precision": rng.choice(["fp64", "fp32"])}


# ------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=4)
def _mesh(scene, size, variant):
    """A seeded scene's geometry and materials (host arrays)."""
    if scene == "strip":
        return scenes.reference_main_scene().scene
    if scene == "site":
        return scenes.small_scene(seed=0x5B5 + variant).scene
    if scene == "canyon":  # the ground and the first `size` of its 400 boxes
        sc = scenes.urban_scene(seed=0x5B6 + variant, rx_pitch=500.0).scene
        n = 2 + 12 * size
        return scenes.Scene(sc.name, sc.tri[:n], sc.normal[:n], sc.material_id[:n], sc.materials)
    return scenes.large_scene(seed=0x5B8 + variant, n_rx=1, cells=size,
                              n_poly=2000 * size * size // (512 * 512)).scene


def _materials(sc, walls):
    """The scene's materials; slab walls get thicknesses of 0.5, 0.2 and 0.01 m
    (ground, concrete, glass)."""
    if walls != "slab":
        return [api.MaterialProperties(*m) for m in sc.materials]
    return [api.MaterialProperties(*m[:6], w) for m, w in zip(sc.materials, (0.5, 0.2, 0.01))]


def _device_scene(sc, walls):
    return api.DeviceScene(api.Mesh(sc.tri, sc.normal, sc.material_id), _materials(sc, walls))


def _spread(rng, n, x0, x1, y0, y1):
    """n points of [x0, x1] x [y0, y1]: a square grid where n is a square (moved
    by part of its pitch), scattered otherwise."""
    m = math.isqrt(n)
    if m * m == n and m > 4:
        u = (np.arange(m) + rng.uniform(0.3, 0.7)) / m
        return np.array([(x0 + (x1 - x0) * a, y0 + (y1 - y0) * b) for a in u for b in u])
    return np.column_stack([rng.uniform(x0, x1, n), rng.uniform(y0, y1, n)])


def _places(rng, scene, sc, size, n_rx):
    """Transmitter and receivers: where that scene's users put them."""
    if scene == "strip":  # a mast over the strip's start, receivers along it
        step = rng.uniform(0.9, 1.1)
        rx = np.array([(0.0, step * i, 3.0) for i in range(n_rx)])
        return (float(rng.uniform(-2, 2)), 0.0, float(rng.uniform(4, 6))), rx
    if scene == "site":
        xy = _spread(rng, n_rx, -90.0, 90.0, -90.0, 90.0)
        return (float(rng.uniform(-3, 3)), float(rng.uniform(-3, 3)), 10.0), \
            np.column_stack([xy, np.full(n_rx, 1.5)])
    if scene == "canyon":  # over a street crossing; receivers at street level
        xy = _spread(rng, n_rx, -500.0, 500.0, -500.0, 500.0)
        tx = (50.0 * int(rng.integers(-4, 5)), 50.0 * int(rng.integers(-4, 5)),
              float(rng.uniform(15, 30)))
        return tx, np.column_stack([xy, np.full(n_rx, 1.5)])
    half = float(size)  # 2 m cells
    grid = sc.tri[:size * size, 0].reshape(size, size, 3)

    def ground(x, y):
        i = np.clip(((np.asarray(x) + half) / 2.0).astype(int), 0, size - 1)
        j = np.clip(((np.asarray(y) + half) / 2.0).astype(int), 0, size - 1)
        return grid[i, j, 2].astype(np.float64)

    x, y = rng.uniform(-15, 15, 2)
    rxy = rng.uniform(-half + 1, half - 1, (n_rx, 2))
    return (float(x), float(y), float(ground(x, y)) + 30.0), \
        np.column_stack([rxy, ground(rxy[:, 0], rxy[:, 1]) + 1.5])


_FREQUENCY = {"strip": 1.8e9, "site": 2.4e9, "canyon": 28e9, "terrain": 3.5e9}
# the reference's main() points the dipole along y; elsewhere z is up
_FRAME = {"strip": (0, 1, 0, 0, 0, 1, 1, 0, 0)}


def _request(case, tx, rx):
    slab = case["walls"] == "slab"
    frame = scenes.ROTATED_TX_FRAME if slab else \
        _FRAME.get(case["scene"], (1, 0, 0, 0, 1, 0, 0, 0, 1))
    return api.make_request(tx, frame, case["reflections"], case["transmissions"],
                            _FREQUENCY[case["scene"]], 1.0, not slab, rx, case["level"],
                            antenna=case["antenna"], precision=case["precision"])


def _inputs(case, seed):
    """(scene geometry, transmitter, receivers) of a trace or solve case."""
    rng = np.random.default_rng([seed, 11])
    sc = _mesh(case["scene"], case["size"], 0)
    return (sc, *_places(rng, case["scene"], sc, case["size"], case["receivers"]))


def _burst_receivers(case, i):
    part = (7 * i % case["requests"]) / max(1, case["requests"] - 1)
    return int(round(100 * (case["receivers_max"] / 100) ** part))


def _path_fields(case, seed):
    """Path list of a field sum: receivers with skewed path counts (most a few,
    some hundreds), (launch, tree position) ranks, decaying amplitudes."""
    rng = np.random.default_rng([seed, 12])
    n, m = case["paths"], case["receivers"]
    w = rng.pareto(1.5, m) + 0.05
    w = np.minimum(w, 600.0 * w.sum() / n)  # at most some hundred paths on one receiver
    recv = rng.choice(m, n, p=w / w.sum()).astype(np.int32)
    launch = rng.choice(max(n, 1 << 22), n, replace=False).astype(np.int64)
    rank = launch << 17 | rng.integers(1, 1 << 7, n)
    field = rng.normal(size=(n, 6)) * np.exp(rng.uniform(-12, 0, (n, 1)))
    return recv, rank, field


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "sum":
        recv, rank, field = _path_fields(case, seed)
        st["recv"] = torch.from_numpy(recv).cuda()
        st["rank"] = torch.from_numpy(rank).cuda()
        st["field"] = torch.from_numpy(field).cuda()
        st["out"] = torch.empty((case["receivers"], 6), dtype=torch.float64, device="cuda")
        st["precision"] = {"fp64": 0, "fp32": 1}[case["precision"]]
        return st
    if kind == "scene":  # another seed is another model
        sc = _mesh(case["scene"], case["size"], 0)
        shift = np.random.default_rng([seed, 13]).uniform(-0.4, 0.4, 2)
        tri = sc.tri.copy()
        tri[..., 2] *= np.float32(1.0 + 0.5 * shift[0])  # relief and heights scaled
        tri[..., 0] *= np.float32(1.0 + 0.5 * shift[1])
        e = tri.astype(np.float64)
        n = np.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        st["mesh"] = api.Mesh(tri, n.astype(np.float32), sc.material_id)
        st["materials"] = _materials(sc, "fresnel")
        return st
    if kind == "study":
        rng = np.random.default_rng([seed, 14])
        sc = _mesh(case["scene"], case["size"], 1 + seed % 100003)
        tx, rx = _places(rng, case["scene"], sc, case["size"], case["receivers"])
        st["mesh"] = api.Mesh(sc.tri, sc.normal, sc.material_id)
        st["materials"] = _materials(sc, case["walls"])
        st["request"] = _request(case, tx, rx)
        return st
    if kind == "trace":
        sc, tx, rx = _inputs(case, seed)
        bvh = api.BVH()
        st["mesh"] = api.Mesh(sc.tri, sc.normal, sc.material_id)
        bvh.ConstructBVH(st["mesh"])
        st["solver"] = api.RTSolver(api.GlobalConfig(antennaType=case["antenna"],
                                                     fieldPrecision=case["precision"]))
        st["solver"].Init(_materials(sc, case["walls"]), len(sc.materials), bvh)
        st["args"] = (tx, np.array(_FRAME[case["scene"]], float).reshape(3, 3), case["reflections"],
                      case["transmissions"], _FREQUENCY[case["scene"]], 1.0, True, rx, st["mesh"],
                      case["level"])
        return st
    if kind == "solve":
        sc, tx, rx = _inputs(case, seed)
        st["scene"] = _device_scene(sc, case["walls"])
        # paths a receiver may have on average (site: many, in file order)
        st["per_rx"] = 32 if case["scene"] == "site" else 2
        if case["scene"] == "site":  # its caller's triangle vector stays in file order
            st["scene"].set_mesh_order(np.arange(len(sc.tri), dtype=np.int32))
        st["request"] = _request(case, tx, rx)
        return st
    # batch and serve: requests of mixed levels and patterns
    rng = np.random.default_rng([seed, 15])
    canyon = _mesh("canyon", case["size"], 0)
    if kind == "batch":
        _, rx = _places(rng, "canyon", canyon, case["size"], case["receivers"])
        st["scene"] = _device_scene(canyon, "fresnel")
        st["requests"] = []
        for i in range(case["requests"]):
            tx, _ = _places(rng, "canyon", canyon, case["size"], 1)
            q = _solve("", "canyon", case["level_min"] + i % (case["level_max"] - case["level_min"] + 1),
                       case["reflections"], 0, len(rx), antenna=int(rng.integers(0, 3)))
            st["requests"].append(_request(q, tx, rx))
        return st
    site = _mesh("site", 0, 0)
    st["scenes"] = [_device_scene(site, "fresnel"), _device_scene(canyon, "fresnel")]
    st["server"] = api.Server(st["scenes"], slots=case["slots"])
    st["requests"] = []
    for i in range(case["requests"]):
        k = i % 2
        name, sc = (("site", site), ("canyon", canyon))[k]
        # the mix is the case's (receivers spread over their logarithm), its
        # places and patterns the seed's
        n_rx = _burst_receivers(case, i)
        tx, rx = _places(rng, name, sc, case["size"], n_rx)
        q = _solve("", name, case["level_min"] + i // 2 % (case["level_max"] - case["level_min"] + 1),
                   2 + i % 5, 0, n_rx, antenna=int(rng.integers(0, 3)))
        st["requests"].append((k, _request(q, tx, rx)))
    return st


# ------------------------------------------------------------------ one pass


_PER_RAY = ("tri", "cop", "kind", "points")


def _fixed(paths, n_rx, per_rx):
    """Every path in arrays whose length depends on the receivers alone (the
    number of paths differs from place to place): the paths, then zeros."""
    cap = per_rx * n_rx + 4096
    out = {}
    for k, v in paths.items():
        a = np.zeros((3 * cap if k in _PER_RAY else cap, *v.shape[1:]), v.dtype)
        if len(v) > len(a):
            raise RuntimeError(f"{len(v)} {k} values of paths: more than {len(a)}")
        a[:len(v)] = v
        out[k] = a
    return out


def _result(res, per_rx=2):
    """A solve's outputs: fields, their stated bound, every path."""
    out = {"field": res.field, "bound": res.field_bound, "segments": res.counts["segments"],
           "n_paths": res.counts["paths"]}
    paths = res.paths if isinstance(res.paths, dict) else _NO_PATHS
    out["paths"] = _fixed(paths, len(res.field), per_rx)
    return out


_NO_PATHS = {**{k: np.zeros(0, np.int32) for k in ("request", "receiver", "heap", "n_rays",
                                                    "near_edge", "tri", "cop", "kind")},
             **{k: np.zeros(0, np.int64) for k in ("launch", "ray_offset")},
             "field": np.zeros((0, 6)), "points": np.zeros((0, 6))}


def run(st):
    kind = st["kind"]
    if kind == "solve":
        return _result(api.solve(st["scene"], st["request"], with_paths="arrays"), st["per_rx"])
    if kind == "trace":
        st["solver"].ExecuteRayTracing(*st["args"])
        return _result(st["solver"].result)
    if kind == "batch":
        return _result(api.solve(st["scene"], st["requests"], with_paths="arrays"))
    if kind == "serve":
        server, left, done = st["server"], len(st["requests"]), {}
        for tag, (scene, q) in enumerate(st["requests"]):
            server.submit(scene, q, tag)
        while left:
            for item in server.poll(timeout_ms=50, with_paths="arrays"):
                if item["status"]:
                    raise RuntimeError(f"request {item['tag']}: status {item['status']}")
                done[item["tag"]] = item["result"]
                left -= 1
        results = [done[t] for t in range(len(done))]
        each = [r.paths if isinstance(r.paths, dict) else _NO_PATHS for r in results]
        field = np.concatenate([r.field for r in results])
        return {"field": field, "segments": np.array([r.counts["segments"] for r in results]),
                "n_paths": np.array([r.counts["paths"] for r in results]),
                "paths": _fixed({k: np.concatenate([p[k] for p in each]) for k in _NO_PATHS},
                                len(field), 2)}
    if kind == "study":
        scene = api.DeviceScene(st["mesh"], st["materials"])
        out = _result(api.solve(scene, st["request"], with_paths="arrays"))
        scene.close()
        return out
    if kind == "scene":
        scene = api.DeviceScene(st["mesh"], st["materials"])
        out = {"mesh_order": scene.mesh_order(), "coplanar": scene.coplanar_ids()}
        scene.close()
        return out
    lib, ptr = _lib.load(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(lib.sbr_receiver_field_sum_noalloc(
        ptr(st["recv"]), ptr(st["rank"]), ptr(st["field"]), st["recv"].numel(), st["out"].shape[0],
        st["precision"], ptr(st["out"]), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return st["out"]


def work(case):
    """What a pass cannot do without.  Bytes: launch directions (24), triangles
    (48) and receivers (24) read once, a field and its bound per receiver
    (56) written.  Flops: one triangle test (about 60) per launch ray, the
    fewest any closest-hit search runs, and per receiver one reception test
    (about 40)."""
    def rays(level):
        return 10 * 4 ** level + 2

    kind = case["kind"]
    if kind == "sum":
        return {"bytes": 60 * case["paths"] + 48 * case["receivers"], "flops": 6 * case["paths"]}
    if kind == "scene":
        n = 2 * case["size"] ** 2 if case["scene"] == "terrain" else 2 + 12 * case["size"]
        return {"bytes": (52 + 8) * n, "flops": 100 * n}
    tri = {"strip": 2, "site": 122, "canyon": 2 + 12 * case["size"],
           "terrain": 2 * case["size"] ** 2}[case.get("scene", "canyon")]
    if kind in ("batch", "serve"):
        span = case["level_max"] - case["level_min"] + 1
        if kind == "batch":
            levels = [case["level_min"] + i % span for i in range(case["requests"])]
            n_rx = case["requests"] * case["receivers"]
        else:
            levels = [case["level_min"] + i // 2 % span for i in range(case["requests"])]
            n_rx = sum(_burst_receivers(case, i) for i in range(case["requests"]))
        launch = sum(rays(v) for v in levels)
    else:
        launch, n_rx = rays(case["level"]), case["receivers"]
    return {"bytes": 24 * launch + 48 * tri + 80 * n_rx, "flops": 60 * launch + 40 * n_rx}


# ------------------------------------------------------------------ 64 bits


def exact(case, seed):
    """Fields in plain FP64 numpy: of the reflection-only solves on the strip
    and the site (every ray against every triangle; canyon and terrain would
    take minutes to hours), and the field sums."""
    if case["kind"] == "sum":
        recv, rank, field = _path_fields(case, seed)
        order = np.lexsort((rank, recv))
        out = np.zeros((case["receivers"], 6))
        np.add.at(out, recv[order], field[order])
        return out
    if case["kind"] not in ("trace", "solve") or case["scene"] not in ("strip", "site"):
        return None
    if case["transmissions"] or case["walls"] != "fresnel" or case["level"] > 6 or \
            (10 * 4 ** case["level"] + 2) * case["receivers"] * (case["reflections"] + 1) > 3e7:
        return None
    sc, tx, rx = _inputs(case, seed)
    frame = _FRAME.get(case["scene"], (1, 0, 0, 0, 1, 0, 0, 0, 1))
    return {"field": _image_method(sc, np.array(tx), rx, case, np.array(frame, float).reshape(3, 3),
                                   _FREQUENCY[case["scene"]])}


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _launch_directions(level):
    """Vertices of the icosahedron, each face split in four `level` times, in
    the order of their creation."""
    a, b = .525731112119133606, .850650808352039932
    v = [np.array(p) for p in (
        (-a, 0, b), (a, 0, b), (-a, 0, -b), (a, 0, -b), (0, b, a), (0, b, -a), (0, -b, a),
        (0, -b, -a), (b, a, 0), (-b, a, 0), (b, -a, 0), (-b, -a, 0))]
    faces = [(0, 4, 1), (0, 9, 4), (9, 5, 4), (4, 5, 8), (4, 8, 1), (8, 10, 1), (8, 3, 10),
             (5, 3, 8), (5, 2, 3), (2, 7, 3), (7, 10, 3), (7, 6, 10), (7, 11, 6), (11, 0, 6),
             (0, 1, 6), (6, 1, 10), (9, 0, 11), (9, 11, 2), (9, 2, 5), (7, 2, 11)]
    for _ in range(level):
        mids, split = {}, []
        for f in faces:
            m = []
            for i, j in ((f[0], f[1]), (f[1], f[2]), (f[2], f[0])):
                key = (min(i, j), max(i, j))
                if key not in mids:
                    mids[key] = len(v)
                    v.append(_unit(v[i] + v[j]))
                m.append(mids[key])
            split += [(f[0], m[0], m[2]), (f[1], m[1], m[0]), (f[2], m[2], m[1]), tuple(m)]
        faces = split
    return _unit(np.array(v))


def _crossing(v1, e1, e2, o, d):
    """Distance parameter of lines o + t d through triangles (inf: none);
    arrays broadcast over leading axes."""
    eps = float(np.finfo(np.float32).eps)
    h = np.cross(d, e2)
    a = (e1 * h).sum(-1)
    with np.errstate(divide="ignore", invalid="ignore"):
        f = 1.0 / a
        s = o - v1
        u = f * (s * h).sum(-1)
        q = np.cross(s, e1)
        w = f * (d * q).sum(-1)
        t = f * (e2 * q).sum(-1)
        ok = (np.abs(a) >= eps) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > eps)
    return np.where(ok, t, np.inf)


def _coplanar(tri, normal):
    """Group of each triangle: connected over shared edges of equal or opposite
    facet normals."""
    root = list(range(len(tri)))

    def find(i):
        while root[i] != i:
            i = root[i]
        return i

    edges = {}
    for i, t in enumerate((tri + np.float32(0.0)).tolist()):
        c = [tuple(p) for p in t]
        for p, q in ((0, 1), (1, 2), (2, 0)):
            edges.setdefault(frozenset((c[p], c[q])), []).append(i)
    for members in edges.values():
        for j in members[1:]:
            for i in members:
                if i < j and (np.array_equal(normal[i], normal[j]) or
                              np.array_equal(normal[i], -normal[j])):
                    root[max(find(i), find(j))] = min(find(i), find(j))
    return [find(i) for i in range(len(tri))]


def _image_method(sc, tx, rx, case, frame, frequency):
    """Received fields (n_rx, 3): rays traced over reflections, captured by the
    first segment whose reception sphere holds the receiver, corrected by the
    image method, one path kept per sequence of coplanar groups, fields summed."""
    tri = sc.tri.astype(np.float64)
    v1, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = sc.normal.astype(np.float64)
    group = _coplanar(sc.tri, sc.normal)
    d = _launch_directions(case["level"])
    live = np.arange(len(d))
    o = np.broadcast_to(tx, d.shape).copy()
    total = np.zeros(len(d))   # length up to the segment
    unfold = np.zeros(len(d))  # the reference's capture length: sum of those so far
    seq = np.zeros((len(d), 0), int)
    tan_beta = math.tan(math.acos(-1.0 / math.sqrt(5.0)) / (3.0 * (case["level"] + 1)))
    todo = [np.ones(len(d), bool) for _ in rx]  # launches that have not captured receiver k
    found = [{} for _ in rx]  # (triangle sequence) -> first launch
    for depth in range(case["reflections"] + 1):
        best, hit = np.full(len(d), np.inf), np.full(len(d), -1)
        for i in range(0, len(d), 4096):
            b = slice(i, i + 4096)
            t = _crossing(v1[None], e1[None], e2[None], o[b, None], d[b, None])
            hit[b] = t.argmin(1)
            best[b] = t.min(1)
        miss = ~np.isfinite(best)
        far = 1e10 if depth == 0 else 1e2
        end = o + np.where(miss, far, best)[:, None] * d
        for k, c in enumerate(rx):
            seg = end - o
            lam = (seg * (c - o)).sum(1) / (seg * seg).sum(1)
            p = o + np.minimum(lam, 1.0)[:, None] * seg
            got = (lam >= 0) & todo[k][live] & \
                (np.linalg.norm(c - p, axis=1) <= (unfold + np.linalg.norm(p, axis=1)) * tan_beta)
            for i in np.flatnonzero(got):
                key = tuple(seq[i])
                found[k].setdefault(key, int(live[i]))
            todo[k][live[got]] = False
        keep = ~miss
        live, hit, p, d = live[keep], hit[keep], end[keep], d[keep]
        total, unfold, seq = total[keep], unfold[keep], seq[keep]
        total = total + np.linalg.norm(p - o[keep], axis=1)
        unfold = unfold + total
        seq = np.column_stack([seq, hit])
        d = _unit(d - 2.0 * n[hit] * (n[hit] * d).sum(1)[:, None])
        o = p
    out = np.zeros((len(rx), 3), complex)
    for k, c in enumerate(rx):
        seen = set()
        for key, _ in sorted(found[k].items(), key=lambda kv: kv[1]):
            if not key:  # direct: nothing in between
                t = _crossing(v1, e1, e2, tx, c - tx).min()
                pts = [tx, c] if not t < 1.0 else None
            else:
                img = [tx]
                for s in key:
                    img.append(img[-1] - 2.0 * np.dot(n[s], img[-1] - v1[s]) * n[s])
                pts, target = [c], c
                for s, im in zip(key[::-1], img[:0:-1]):
                    t = _crossing(v1[s], e1[s], e2[s], im, target - im)
                    if not np.isfinite(t):
                        pts = None
                        break
                    target = im + t * (target - im)
                    pts.append(target)
                if pts is not None:
                    pts = [tx] + pts[::-1]
            marks = tuple(group[s] for s in key)
            if pts is None or marks in seen:
                continue
            seen.add(marks)
            out[k] += _path_field(sc, pts, key, case["antenna"], frame, frequency, tri, n)
    return out


def _path_field(sc, pts, key, antenna, frame, frequency, tri, n):
    """Field of one reflected path of 1 W, segment by segment in the spherical
    basis of the frame it starts in."""
    c0, mu0 = 2.99792458e8, 4e-7 * math.pi
    e0, eta0 = 1.0 / (mu0 * c0 * c0), mu0 * c0
    field, length = np.zeros(3, complex), 0.0
    for i in range(len(pts) - 1):
        if i == 0:
            cur = frame
        else:
            s = key[i - 1]
            y = _unit(tri[s, 1] - tri[s, 0])
            cur = np.array([np.cross(y, n[s]), y, n[s]])
        seg = pts[i + 1] - pts[i]
        loc = cur @ seg
        length += np.linalg.norm(loc)
        th = math.atan2(math.hypot(loc[0], loc[1]), loc[2])
        ph = math.atan2(loc[1], loc[0])
        st, ct, sp, cp = math.sin(th), math.cos(th), math.sin(ph), math.cos(ph)
        basis = np.array([[st * cp, ct * cp, -sp], [st * sp, ct * sp, cp], [ct, -st, 0.0]])
        if i == 0:
            inc = np.zeros(3, complex)
            if antenna == 0:
                inc[0] = 1j * math.sqrt(60.0)
            elif antenna == 1:
                inc[1] = 1j * math.sqrt(90.0) * st
            else:
                inc[1] = 1j * math.sqrt(60.0) * (math.cos(math.pi * ct / 2.0) / st)
        else:
            inc = basis.T @ (cur.T @ field)
            a, b = _unit(seg), _unit(cur[2])
            x = float(np.dot(a, b))
            ang = math.pi - 2.0 * math.asin(np.linalg.norm(a + b) / 2.0) if x < 0 else \
                2.0 * math.asin(np.linalg.norm(a - b) / 2.0)
            m = sc.materials[int(sc.material_id[key[i - 1]])]
            nt = np.sqrt(complex(m[3], -m[5] / (e0 * 2.0 * math.pi * frequency)))
            cos_i, cos_t = math.cos(ang), np.cos(np.arcsin(math.sin(ang) / nt))
            eta_t = eta0 / nt
            tm = (eta0 * cos_i - eta_t * cos_t) / (eta0 * cos_i + eta_t * cos_t)
            te = -(eta_t / cos_t - eta0 / cos_i) / (eta_t / cos_t + eta0 / cos_i)
            inc = inc * np.array([1.0, tm, te])
        field = cur.T @ (basis @ inc)
    k = 2.0 * math.pi / (c0 / frequency)
    return field * np.exp(-1j * k * length) / length
