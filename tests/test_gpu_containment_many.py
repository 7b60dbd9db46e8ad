"""Containment rays that cross more triangles than a warp's list holds (512): objects crossed once,
twice and hundreds of times each, more objects than the list has room for, ids below zero, and
boxes that all lie on the ray, which no stack holds at once.  Pairs equal the CPU oracle's, the
counters what the geometry says, and the time stays near that of rays the list holds."""
import ctypes
import time

import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _nested(k):
    """k concentric cubes: a ray from the centre crosses each once, and each contains it."""
    return [(np.full(3, -1.0 - 0.01 * j), np.full(3, 1.0 + 0.01 * j)) for j in range(k)]


def _stacked(k):
    """k boxes above the origin, crossed twice each."""
    return [(np.array([-1.0, -1.0, 50.0 + j]), np.array([1.0, 1.0, 50.5 + j])) for j in range(k)]


def _sources(n):
    c = np.random.default_rng(3).uniform(-0.4, 0.4, (n, 3))
    return synth.box_set([(p - 0.05, p + 0.05) for p in c], edges=False)


def _target(boxes, objects=None):
    """The boxes' objects in a mixed order, or the given ids."""
    g = synth.box_set(boxes, edges=False)
    ids = np.random.default_rng(len(boxes)).permutation(len(boxes)) if objects is None else np.asarray(objects)
    return synth.make_geometry(g.vertices, g.indices, ids[g.tri2obj], edges=False)


CASES = {"540 nested": (lambda: _target(_nested(540)), 540, 540),
         "3000 nested": (lambda: _target(_nested(3000)), 3000, 3000),
         "257 stacked": (lambda: _target(_stacked(257)), 514, 257),
         "1500 stacked in 20": (lambda: _target(_nested(20) + _stacked(1500)), 3020, 1520),
         "one of 700 boxes among 600": (lambda: _target(_nested(600) + _stacked(700), [*range(600)] + [77] * 700), 2000, 600),
         "two of 401 each": (lambda: _target(_nested(802), [5, 9] * 401), 802, 2)}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("n", [1, 50])
def test_pairs_and_counters(cuda, name, n):
    make, crossings, candidates = CASES[name]
    A, B = _sources(n), make()
    b, src = api.Bvh(api.DeviceGeometry(B)), api.DeviceGeometry(A)
    want = np.sort(bind.containment(A, B.vertices, B.indices, B.tri2obj))
    L = _lib.load()
    for track in (0, 1):
        ps = api.PairSet(1 << 18)
        L.rs_pairset_set_tracking(ps.handle, track)
        api.containment(b, src, ps)
        np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)
        if track:
            c = (ctypes.c_uint64 * 8)()
            assert L.rs_pairset_counters(ps.handle, c, None) == 0
            assert list(c)[4:7] == [n, n * crossings, n * candidates]


def test_an_id_below_zero(cuda):
    A, B = _sources(3), _target(_nested(600), [-1, 4] * 300)
    B = synth.make_geometry(B.vertices, B.indices, np.where(np.arange(len(B.indices)) < 12, 4, B.tri2obj), edges=False)
    ps = api.PairSet(1 << 10)  # 4 is crossed 301 times, -1 299 times
    api.containment(api.Bvh(api.DeviceGeometry(B)), api.DeviceGeometry(A), ps)
    got = {tuple(p) for p in api.keys_to_pairs(ps.finalize()).tolist()}
    assert got == {(o, t) for o in range(3) for t in (4, -1)}


def test_a_list_that_overflows_costs_no_fallback(cuda):
    src = api.DeviceGeometry(_sources(20000))

    def seconds(k):
        b = api.Bvh(api.DeviceGeometry(_target(_stacked(k))))
        best = np.inf
        ps = api.PairSet(1 << 10)
        for _ in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            api.containment(b, src, ps)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best
    assert seconds(300) < 10 * seconds(200)  # 36 times, by the one-thread passes


@pytest.mark.parametrize("n", [65536, 65537, 70003])
def test_more_objects_than_warps(cuda, n):
    """Around the number from which rays go in packets: columns of 3, 9 and 12 boxes, one of 520 nested,
    one beside everything, an object in seven without a triangle."""
    column = np.arange(n) % 5
    c = np.random.default_rng(n).uniform(-0.4, 0.4, (n, 3)) + np.stack([100.0 * column, 0 * column, 0 * column], 1)
    # one triangle an object: its first vertex is the ray's origin
    V = (c[:, None] + np.array([[0, 0, 0], [0.01, 0, 0], [0, 0.01, 0.01]])).astype(np.float32).reshape(-1, 3)
    keep = np.arange(n) % 7 != 3
    keep[-1] = True
    I = np.arange(3 * n).reshape(-1, 3)[keep]
    A = synth.make_geometry(V, I, np.arange(n)[keep], edges=False)
    at = lambda boxes, k: [(lo + [100.0 * k, 0, 0], hi + [100.0 * k, 0, 0]) for lo, hi in boxes]
    B = _target(at(_nested(3), 0) + at(_nested(1) + _stacked(4), 1) + at(_nested(12), 2) + at(_nested(520), 3))
    ps = api.PairSet(1 << 24)
    L = _lib.load()
    L.rs_pairset_set_tracking(ps.handle, 1)
    api.containment(api.Bvh(api.DeviceGeometry(B)), api.DeviceGeometry(A), ps)
    want = np.sort(bind.containment(A, B.vertices, B.indices, B.tri2obj))
    np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)
    per = np.bincount(column[keep], minlength=5)
    c = (ctypes.c_uint64 * 8)()
    assert L.rs_pairset_counters(ps.handle, c, None) == 0
    assert list(c)[4:7] == [keep.sum(), int(per @ [3, 9, 12, 520, 0]), int(per @ [3, 5, 12, 520, 0])]


def test_many_short_rays_fill_their_warps(cuda):
    """Objects below three large ones: 80,000, in packets first, take less time than 60,000, a warp each."""
    from rayspace3d_gb300 import gen
    target = api.Bvh(gen.instanced_set(3, 6, 40.0, 50.0, 100.0, seed=6))

    def seconds(n):
        src = gen.instanced_set(n, 0, 0.05, 0.2, 100.0, seed=5)
        ps, best = api.PairSet(1 << 20), np.inf
        for _ in range(20):
            torch.cuda.synchronize()
            t = time.perf_counter()
            api.containment(target, src, ps)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best
    assert seconds(80000) < seconds(60000)  # 0.4 times; all of them a warp each, 1.2 times
