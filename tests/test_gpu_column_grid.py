"""Column grid of axis-aligned point queries where its sizing, lists and lengths change.

A scene of many small objects over a wide area (cells larger than four a triangle), one
triangle pair that covers every cell, stacks of nested objects whose rays cross more
triangles than a point's slots, a warp's and a block's worth hold, and flat or single
meshes.  Object ids and inside bits equal the CPU oracle's.
"""
import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _join(parts):
    Vs, Is, Ts, v0, o0 = [], [], [], 0, 0
    for V, F, T in parts:
        Vs.append(np.asarray(V, np.float32))
        Is.append(np.asarray(F, np.uint32) + np.uint32(v0))
        Ts.append(np.asarray(T, np.int32) + o0)
        v0 += len(V)
        o0 += int(np.max(T)) + 1
    return synth.make_geometry(np.concatenate(Vs), np.concatenate(Is), np.concatenate(Ts), edges=False)


def _nested(k, level, centre, r0, step):
    """k concentric spheres: a ray from the centre crosses k triangles or a few more."""
    v, f = synth.icosphere(level)
    return [((v * (r0 + step * j) + centre).astype(np.float32), f, np.zeros(len(f), np.int32)) for j in range(k)]


def _quad(lo, hi, axis, at):
    u, v = (axis + 1) % 3, (axis + 2) % 3
    V = np.zeros((4, 3))
    V[:, axis] = at
    V[[1, 2], u], V[[0, 3], u] = hi, lo
    V[[2, 3], v], V[[0, 1], v] = hi, lo
    return V.astype(np.float32), np.array([[0, 1, 2], [0, 2, 3]]), np.zeros(2, np.int32)


def _scattered(axis):
    s = synth.sphere_set(3000, 2, 0.2, 1.0, 60.0, np.random.default_rng(7), edges=False)
    parts = [(s.vertices, s.indices, s.tri2obj), _quad(-3.0, 64.0, axis, 31.0)]
    parts += _nested(20, 1, 20.0, 0.5, 0.05) + _nested(60, 1, 30.0, 0.5, 0.02)
    return _join(parts)


def _deep(axis):
    return _join(_nested(9, 2, 0.0, 1.0, 0.07) + _nested(40, 1, 6.0, 1.0, 0.02) + _nested(300, 0, 12.0, 1.0, 0.004))


def _flat(axis):
    v, f = synth.icosphere(2)
    v = v.copy()
    v[:, (axis + 1) % 3] = 0.25  # no extent across the rays on one axis
    return _join([(v, f, np.zeros(len(f), np.int32))])


def _single(axis):
    return _join([_quad(-1.0, 1.0, axis, 0.5)])


def _points(g, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = g.vertices.min(0) - 0.5, g.vertices.max(0) + 0.5
    pts = (lo + rng.random((n, 3)) * (hi - lo)).astype(np.float32)
    k = n // 8
    near = g.vertices[rng.integers(0, len(g.vertices), k)]
    pts[:k] = near  # exactly on vertices
    pts[k:2 * k] = near + rng.normal(0, 0.05, (k, 3)).astype(np.float32)
    b0, b1 = g.vertices.min(0), g.vertices.max(0)  # on the filter box's faces, edges and corners
    pts[-24:] = np.where(rng.random((24, 3)) < 0.4, b0, np.where(rng.random((24, 3)) < 0.6, b1, pts[-24:]))
    for j, c in enumerate((0.0, 6.0, 12.0, 20.0, 30.0)):  # inside the nested objects
        pts[2 * k + 40 * j:2 * k + 40 * (j + 1)] = c + rng.normal(0, 0.3, (40, 3))
    return pts


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("scene", [_scattered, _deep, _flat, _single])
def test_axis_points_match_oracle(cuda, scene, axis):
    g = scene(axis)
    d = [0.0, 0.0, 0.0]
    d[axis] = 1.0
    bvh = api.Bvh(api.DeviceGeometry(g))
    for n in (3001, 1):
        pts = _points(g, n, 11 + axis) if n > 1 else g.vertices[:1].copy()
        for filtered in (False, True):
            want = bind.pim(g.vertices, g.indices, g.tri2obj, pts, direction=tuple(d), filtered=filtered)
            obj, inside = api.point_in_mesh(bvh, torch.from_numpy(pts).cuda(), direction=tuple(d), filtered=filtered)
            got = obj.cpu().numpy()
            bad = np.nonzero(got != want)[0]
            assert len(bad) == 0, f"{len(bad)} differ, first {bad[:5]}: {got[bad[:5]]} against {want[bad[:5]]}"
            assert np.array_equal(inside.cpu().numpy().astype(bool), want >= 0)
