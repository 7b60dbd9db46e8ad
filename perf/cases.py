"""The workloads that the engine's speed is judged by: point queries, joins, preprocessing, batches and the
learned estimator, each through the calls that a user's program makes.

Sizes come from the engine's own configurations (one million and a hundred million points on an icosphere, 10k + 10k
objects in cubes of side 1000 and 80.7, uneven intersection sets, clustered data sets, degenerate batches) or span
the range around them.  Geometry is generated on the device; every edge payload is in the order that a `.pre` file
holds it in (api.extract_edges).
"""
import ctypes
import math

import numpy as np
import torch

from rayspace3d_gb300 import _lib, api, gen, learned

DIRECTIONS = {"x": (1.0, 0.0, 0.0), "y": (0.0, 1.0, 0.0), "z": (0.0, 0.0, 1.0),
              "oblique": (0.36, -0.48, 0.8)}
GRID = 128
HIDDEN = 512
ROOM = 200  # keys an object that a caller's result buffer has room for


def listed():
    return [
        # A service that asks about a few points at a time against a mesh it holds: latency is all there is.
        {"name": "points_small", "kind": "points", "points": 1000, "objects": 1, "level": 2, "direction": "z",
         "filtered": False, "snapped": 0.0, "build": False, "compact": True},
        # The plain point-in-mesh configuration: one million points, +x rays, one inside bit and object a point.
        {"name": "points_1m", "kind": "points", "points": 1000000, "objects": 1, "level": 4, "direction": "x",
         "filtered": False, "snapped": 0.0, "build": False, "compact": False},
        # A point cloud scanned through the bounding-box filter, with points that lie exactly on the mesh (samples
        # of its own surface), and the list of hits that raytracer_filter_refine writes.
        {"name": "points_cloud", "kind": "points", "points": 60000001, "objects": 1, "level": 6, "direction": "z",
         "filtered": True, "snapped": 0.05, "build": False, "compact": True},
        # One run of raytracer on a new scene: the index is built, asked once and the hits are listed.
        {"name": "points_new_scene", "kind": "points", "points": 500009, "objects": 20000, "level": 2,
         "direction": "z", "filtered": False, "snapped": 0.0, "build": True, "compact": True},
        # The smallest join: two small sets, overlap and containment, everything built for it.
        {"name": "join_small", "kind": "join", "objects": 150, "level": 1, "world": 12.0, "containment": True},
        # The headline join: 10k + 10k objects, sparse; built, estimated, joined, sorted.
        {"name": "join_sparse", "kind": "join", "objects": 10000, "level": 2, "world": 1000.0, "containment": False},
        # The same sets at the selectivity of 1e-4: most objects have a partner.
        {"name": "join_dense", "kind": "join", "objects": 10000, "level": 2, "world": 80.7, "containment": False},
        # Full intersection of uneven sets (80 to 20,480 triangles an object), some objects inside others.
        {"name": "join_uneven", "kind": "uneven", "objects": 3001, "world": 621.0},
        # Clustered sets of spheres and boxes, radii 0.1 to 50: the joins that label the estimator's training data.
        {"name": "join_clustered", "kind": "clustered", "objects": 20000, "components": 12},
        # Preprocessing one set: its unique edges and its grid statistics.
        {"name": "preprocess", "kind": "preprocess", "objects": 10000, "level": 2, "world": 1000.0},
        # A server's batch: point queries of mixed size, direction and degeneracy and both directions of some joins
        # in one launch, submitted again and again on the handles it keeps.
        {"name": "batch", "kind": "batch", "queries": 24, "most_points": 400000, "joins": 2, "objects": 3000},
        # The learned estimator: gradients of one minibatch, read by the host, and predictions for held-out pairs.
        {"name": "estimator", "kind": "estimator", "rows": 64, "held_out": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "points", "points", "join", "join", "uneven", "clustered", "preprocess", "batch",
                       "estimator"])
    if kind == "points":
        scene = rng.random() < 0.4
        build = scene and rng.random() < 0.6
        return {"kind": kind, "points": _log(rng, 1000, 5e5 if scene else 5e7),
                "objects": _log(rng, 30, 20000) if scene else 1,
                "level": rng.randint(0, 2) if scene else rng.randint(1, 6),
                "direction": rng.choice(["x", "y", "z", "z"]), "filtered": rng.random() < 0.3,
                "snapped": rng.choice([0.0, 0.0, 0.05]), "build": build, "compact": rng.random() < 0.6}
    if kind == "join":
        n = _log(rng, 100, 10000)
        # between the two densities of the 10k sets
        side = math.exp(rng.uniform(math.log(80.7), math.log(1000.0)))
        return {"kind": kind, "objects": n, "level": rng.randint(1, 2),
                "world": round(side * (n / 10000.0) ** (1.0 / 3.0), 3), "containment": rng.random() < 0.3}
    if kind == "uneven":
        n = _log(rng, 100, 3000)
        return {"kind": kind, "objects": n, "world": round(2000.0 * (n / 100000.0) ** (1.0 / 3.0), 3)}
    if kind == "clustered":
        return {"kind": kind, "objects": _log(rng, 300, 20000), "components": rng.randint(8, 24)}
    if kind == "preprocess":
        return {"kind": kind, "objects": _log(rng, 20, 10000), "level": rng.randint(1, 2),
                "world": round(rng.uniform(200.0, 1000.0), 2)}
    if kind == "batch":
        return {"kind": kind, "queries": rng.randint(4, 24), "most_points": _log(rng, 20000, 400000),
                "joins": rng.randint(1, 3), "objects": _log(rng, 300, 3000)}
    return {"kind": "estimator", "rows": rng.randint(8, 96), "held_out": rng.randint(40, 1000)}


def _here():
    return torch.cuda.current_stream().cuda_stream


def _filled(n, dtype, count=1):
    """The caller's own result buffers, -1 beyond the results."""
    return [torch.full((n,), -1, dtype=dtype, device="cuda") for _ in range(count)]


def _in_file_order(dg):
    """The geometry with its edge payload as a `.pre` file holds it."""
    edges = tuple(t.clone() for t in api.extract_edges(dg.V, dg.I, dg.T))
    return api.DeviceGeometry.from_tensors(dg.V, dg.I, dg.T, edges=edges)


def _cell_volume(world):
    c = np.float32(np.float32(world) / np.float32(GRID))
    return float(np.float32(np.float32(c * c) * c))


def _cells(dg, objects, world):
    """The 128^3 grid statistics of a set, as its `.pre` file holds them."""
    cells = torch.empty(GRID ** 3 * 16, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().rs_grid_stats(dg.V.data_ptr(), dg.nV, dg.I.data_ptr(), dg.nF, dg.T.data_ptr(), objects,
                                         GRID, float(world), cells.data_ptr(), None,
                                         _here()), "rs_grid_stats")
    return cells


def _with_grid(dg, objects, world):
    dg = _in_file_order(dg)
    dg.cells = _cells(dg, objects, world)
    return dg


def _scene_side(objects):
    """The cube that gives 20,000 objects of radius 0.5 to 2 a filling of about a tenth."""
    return 2.0 + 2.0 * 40.0 * (objects / 20000.0) ** (1.0 / 3.0)


def prepare(case, seed):
    return {"points": _prepare_points, "join": _prepare_join, "uneven": _prepare_uneven,
            "clustered": _prepare_clustered, "preprocess": _prepare_preprocess, "batch": _prepare_batch,
            "estimator": _prepare_estimator}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


# ---- points

def _prepare_points(case, seed):
    if case["objects"] == 1:
        mesh = gen.instanced_set(1, case["level"], 1.0, 1.0, 0.0, seed=2 * seed)
        pad = 0.5
    else:
        mesh = gen.instanced_set(case["objects"], case["level"], 0.5, 2.0, _scene_side(case["objects"]), seed=2 * seed)
        pad = 0.25
    pts = gen.mesh_points(mesh, case["points"], seed=2 * seed + 1, frac_snapped=case["snapped"], pad=pad)
    return {"run": _run_points, "mesh": mesh, "points": pts, "direction": DIRECTIONS[case["direction"]],
            "filtered": case["filtered"], "hits": _filled(case["points"], torch.int32, 2) if case["compact"] else None,
            "bvh": None if case["build"] else api.Bvh(mesh)}


def _run_points(s):
    bvh = s["bvh"] if s["bvh"] is not None else api.Bvh(s["mesh"])
    obj, inside = api.point_in_mesh(bvh, s["points"], direction=s["direction"], filtered=s["filtered"])
    if s["hits"] is None:
        return obj, inside
    ids, objs = s["hits"]
    count = ctypes.c_uint64()
    _lib.check(_lib.load().rs_compact_hits(obj.data_ptr(), obj.numel(), ids.data_ptr(), objs.data_ptr(), ids.numel(),
                                           ctypes.byref(count), _here()), "rs_compact_hits")
    return obj, inside, ids, objs, count.value


# ---- joins

def _prepare_join(case, seed):
    n, w = case["objects"], case["world"]
    A = _with_grid(gen.instanced_set(n, case["level"], 0.5, 2.0, w, seed=2 * seed), n, w)
    B = _with_grid(gen.instanced_set(n, case["level"], 0.5, 2.0, w, seed=2 * seed + 1), n, w)
    return _join_state(A, B, n, w, case["containment"])


def _prepare_uneven(case, seed):
    n, w = case["objects"], case["world"]
    A, B, _ = gen.intersection_sets(n, seed, world=w)
    return _join_state(_with_grid(A, n, w), _with_grid(B, n, w), n, w, True)


def _boxes_of(case):
    return case["objects"] // 4


def _prepare_clustered(case, seed):
    n, boxes = case["objects"], _boxes_of(case)

    def side(k):
        centers = gen.mixture_centers(n, case["components"], learned.WORLD, k)
        parts = [gen.instanced_set(n - boxes, 1, 0.1, 50.0, learned.WORLD, seed=k + 1, centers=centers[:n - boxes]),
                 gen.instanced_set(boxes, 0, 0.1, 50.0, learned.WORLD, seed=k + 2, kind="box",
                                   centers=centers[n - boxes:])]
        return _with_grid(gen.concat(parts), n, learned.WORLD)

    return _join_state(side(8 * seed), side(8 * seed + 4), n, learned.WORLD, False)


def _join_state(A, B, objects, world, containment):
    return {"run": _run_join, "A": A, "B": B, "volume": _cell_volume(world), "containment": containment,
            "keys": _filled(ROOM * objects, torch.int64)[0], "streams": (torch.cuda.Stream(), torch.cuda.Stream())}


def _run_join(s):
    A, B = s["A"], s["B"]
    here = torch.cuda.current_stream()
    for side in s["streams"]:
        side.wait_stream(here)
    a = api.Bvh(A, stream=s["streams"][0], asynchronous=True)
    b = api.Bvh(B, stream=s["streams"][1], asynchronous=True)
    raw, means = api.estimate_grid(A.cells, B.cells, GRID ** 3, s["volume"])
    estimate = int(_lib.load().rs_estimate_pairs_from_raw(raw, (ctypes.c_float * 4)(*means), s["volume"], 1))
    pairs = api.PairSet(api.hash_size_pow2(estimate))
    api.overlap_join(a, b, pairs, with_containment=s["containment"])
    count = _sorted_keys(pairs, 1, s["keys"], _here())
    for handle in (a, b, pairs):
        handle.close()
    return s["keys"], count, estimate


def _sorted_keys(pairs, order, keys, stream):
    """The sorted keys into the caller's buffer, in stream order, as PairSet.finalize does into its own."""
    count = ctypes.c_uint64()
    _lib.check(_lib.load().rs_pairset_finalize(pairs.handle, order | api.RS_FINALIZE_NO_WAIT, keys.data_ptr(),
                                               keys.numel(), ctypes.byref(count), stream), "rs_pairset_finalize")
    return count.value


# ---- preprocessing

def _prepare_preprocess(case, seed):
    n = case["objects"]
    mesh = gen.instanced_set(n, case["level"], 0.5, 2.0, case["world"], seed=seed)
    return {"run": _run_preprocess, "mesh": mesh, "objects": n, "world": case["world"]}


def _run_preprocess(s):
    m = s["mesh"]
    return api.extract_edges(m.V, m.I, m.T) + (_cells(m, s["objects"], s["world"]),)


# ---- batches

def _batch_points(case, q):
    """Point counts of a batch's queries: spread over the logarithm from 1000 to the most."""
    return int(1000 * (case["most_points"] / 1000.0) ** ((q % 8) / 7.0)) + q


def _batch_level(q):
    return 1 + (q * 5) % 6


def _prepare_batch(case, seed):
    L = _lib.load()
    stream = torch.cuda.Stream()
    h = ctypes.c_void_p()
    _lib.check(L.rs_batch_create(ctypes.byref(h)), "rs_batch_create")
    total = sum(_batch_points(case, q) for q in range(case["queries"]))
    obj = torch.empty(total, dtype=torch.int32, device="cuda")
    inside = torch.empty(total, dtype=torch.uint8, device="cuda")
    keep, at = [], 0
    for q in range(case["queries"]):
        n = _batch_points(case, q)
        mesh = gen.instanced_set(1, _batch_level(q), 1.0, 1.0, 0.0, seed=1000 * seed + q)
        pts = gen.mesh_points(mesh, n, seed=1000 * seed + 500 + q, frac_snapped=0.2)
        bvh = api.Bvh(mesh)
        d = DIRECTIONS[("x", "y", "z", "oblique")[q % 4]]
        _lib.check(L.rs_batch_add_pim(h, bvh.handle, pts.data_ptr(), n, *d, obj[at:].data_ptr(),
                                      inside[at:].data_ptr(), None), "rs_batch_add_pim")
        keep.append((mesh, pts, bvh))
        at += n
    sets = []
    world = 1000.0 * (case["objects"] / 10000.0) ** (1.0 / 3.0)
    for j in range(case["joins"]):
        A, B = (_in_file_order(gen.instanced_set(case["objects"], 2, 0.5, 2.0, world, seed=1000 * seed + 900 + 2 * j + k))
                for k in (0, 1))
        a, b, ps = api.Bvh(A), api.Bvh(B), api.PairSet(1 << 16)
        for target, source, swap in ((b, A, 0), (a, B, 1)):
            _lib.check(L.rs_batch_add_edges(h, target.handle, *source.edge_ptrs(), source.nE, swap, ps.handle, None),
                       "rs_batch_add_edges")
        keep.append((a, b))
        sets.append((ps, _filled(ROOM * case["objects"], torch.int64)[0]))
    torch.cuda.synchronize()
    return {"run": _run_batch, "batch": _Batch(h), "stream": stream, "obj": obj, "inside": inside, "sets": sets,
            "keep": keep}


class _Batch:
    """A batch handle, released with its last reference."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        _lib.load().rs_batch_destroy(self.handle)


def _run_batch(s):
    L, stream = _lib.load(), s["stream"]
    for ps, _ in s["sets"]:
        ps.clear(stream=stream)
    _lib.check(L.rs_batch_submit(s["batch"].handle, stream.cuda_stream), "rs_batch_submit")
    _lib.check(L.rs_batch_wait(s["batch"].handle, None), "rs_batch_wait")
    counts = [_sorted_keys(ps, 0, keys, stream.cuda_stream) for ps, keys in s["sets"]]
    torch.cuda.current_stream().wait_stream(stream)
    return s["obj"], s["inside"], [keys for _, keys in s["sets"]], counts


# ---- the learned estimator

def _parameters(seed):
    """W1, b1, W2, b2, W3, b3 with He-uniform weights, one FP32 array on the device."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3 * seed)
    parts = []
    for out, fan_in in ((HIDDEN, learned.N_FEAT), (HIDDEN, HIDDEN), (1, HIDDEN)):
        bound = math.sqrt(6.0 / fan_in)
        parts.append((torch.rand(out * fan_in, generator=g, device="cuda") * 2 - 1) * bound)
        parts.append((torch.rand(out, generator=g, device="cuda") * 2 - 1) * 0.1)
    return torch.cat(parts)


def _features(case, seed):
    """Minibatch, its targets and held-out rows: pooled grid features are logarithms of counts, half of them zero."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3 * seed + 1)

    def rows(n):
        x = torch.rand((n, learned.N_FEAT), generator=g, device="cuda")
        return torch.where(x < 0.5, torch.zeros_like(x), torch.log1p((x - 0.5) * 40.0)).contiguous()

    X = rows(case["rows"])
    t = torch.randn(case["rows"], generator=g, device="cuda")
    return X, t, rows(case["held_out"])


def _prepare_estimator(case, seed):
    m = learned.Mlp(0)
    m.set_params(_parameters(seed).cpu().numpy())
    X, t, held = _features(case, seed)
    return {"run": _run_estimator, "model": m, "X": X, "t": t, "held": held}


def _run_estimator(s):
    m = s["model"]
    loss = m.gradients(s["X"], s["t"])
    _, gradients = m.params(grads=True)
    return m.forward(s["held"]), gradients, loss


# ---- the least work, and the exact values

def _sphere(level):
    """Vertices, triangles and edges of an icosphere."""
    return 10 * 4 ** level + 2, 20 * 4 ** level, 30 * 4 ** level


def _set_bytes(v, f, e):
    """A set with its edge payload: vertices, indices and objects, endpoints, offsets, counts and sources."""
    return 12 * v + 16 * f + 36 * e


def work(case):
    k = case["kind"]
    if k == "points":
        v, f, _ = (case["objects"] * x for x in _sphere(case["level"]))
        return {"bytes": 17 * case["points"] + 12 * v + 16 * f, "flops": 0}
    grids = 2 * 16 * GRID ** 3
    if k == "join":
        return {"bytes": grids + 2 * _set_bytes(*(case["objects"] * x for x in _sphere(case["level"]))), "flops": 0}
    if k == "uneven":
        mean = [sum(_sphere(level)[i] for level in range(1, 6)) / 5.0 for i in range(3)]
        return {"bytes": grids + 2 * _set_bytes(*(case["objects"] * x for x in mean)), "flops": 0}
    if k == "clustered":
        boxes = _boxes_of(case)
        spheres = [(case["objects"] - boxes) * x for x in _sphere(1)]
        return {"bytes": grids + 2 * _set_bytes(*(s + boxes * x for s, x in zip(spheres, (8, 12, 18)))), "flops": 0}
    if k == "preprocess":
        v, f, e = (case["objects"] * x for x in _sphere(case["level"]))
        return {"bytes": 12 * v + 16 * f + 36 * e + 16 * GRID ** 3, "flops": 0}
    if k == "batch":
        total = 0
        for q in range(case["queries"]):
            v, f, _ = _sphere(_batch_level(q))
            total += 17 * _batch_points(case, q) + 12 * v + 16 * f
        return {"bytes": total + 2 * case["joins"] * _set_bytes(*(case["objects"] * x for x in _sphere(2))), "flops": 0}
    weights = HIDDEN * learned.N_FEAT + HIDDEN * HIDDEN + HIDDEN
    rows = case["rows"] + case["held_out"]
    # weights read, gradients written; the first layer's inputs need no gradient
    return {"bytes": 4 * (2 * weights + rows * (learned.N_FEAT + 1)),
            "flops": 2 * rows * weights + 2 * case["rows"] * (2 * weights - HIDDEN * learned.N_FEAT)}


def exact(case, seed):
    """The estimator's predictions, gradients and loss in 64 bits; every other output is a whole number or a copy."""
    if case["kind"] != "estimator":
        return None
    p = _parameters(seed).double()
    X, t, held = (x.double() for x in _features(case, seed))
    sizes = [HIDDEN * learned.N_FEAT, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN, 1]
    W1, b1, W2, b2, W3, b3 = torch.split(p, sizes)
    W1, W2, W3 = W1.view(HIDDEN, -1), W2.view(HIDDEN, HIDDEN), W3.view(1, HIDDEN)

    def layers(x):
        h1 = torch.relu(x @ W1.T + b1)
        h2 = torch.relu(h1 @ W2.T + b2)
        return h1, h2, (h2 @ W3.T + b3)[:, 0]

    h1, h2, y = layers(X)
    dy = (2.0 / len(t)) * (y - t)
    d2 = dy[:, None] * W3 * (h2 > 0)
    d1 = (d2 @ W2) * (h1 > 0)
    grads = [d1.T @ X, d1.sum(0), d2.T @ h1, d2.sum(0), dy @ h2, dy.sum()]
    return layers(held)[2], torch.cat([g.reshape(-1) for g in grads]), float(((y - t) ** 2).mean())
