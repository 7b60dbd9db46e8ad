"""Unique edges by vertex ranks (rs_extract_edges) at the list lengths where their path
changes: one thread's 32 records and one more, one block's 4096 and one more (the general
path), records staged in shared memory and too many for it, runs of many triangles and
objects on one edge, coinciding and signed-zero vertices, more vertices than corners, and
one position only.  The payload equals the oracle's byte for byte."""
import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import api

pytestmark = pytest.mark.gpu


def _fan(k, rng):
    """k triangles around a hub below all others: its list has 2 k records."""
    a = np.linspace(0.0, 6.0, k + 1)
    V = np.concatenate([[[-5.0, 0.0, 0.0]], np.stack([np.cos(a) + 2, np.sin(a), rng.random(k + 1)], 1)])
    I = np.stack([np.zeros(k, int), np.arange(1, k + 1), np.arange(2, k + 2)], 1)
    return V, I, rng.integers(0, 5, k)


def _book(k, rng):
    """k triangles on one edge, of few objects, both orientations."""
    V = np.concatenate([[[0.0, 0.0, 0.0], [0.0, 0.0, 1.0]], rng.random((k, 3)) + 1])
    I = np.stack([np.zeros(k, int), np.ones(k, int), np.arange(2, k + 2)], 1)
    flip = rng.random(k) < 0.5
    I[flip] = I[flip][:, [1, 0, 2]]
    return V, I, rng.integers(0, 7, k)


def _dense_fans(k, n, rng):
    """n hubs of k triangles each: 2 k records a list over all lists of a block."""
    parts = [_fan(k, rng) for _ in range(n)]
    V = np.concatenate([p[0] + [[20.0 * j, 0, 0]] for j, p in enumerate(parts)])
    I = np.concatenate([p[1] + j * (k + 2) for j, p in enumerate(parts)])
    return V, I, np.repeat(np.arange(n), k)


def _soup(n, rng):
    """Every corner a vertex of its own, few distinct positions (among them -0.0), some
    triangles skipped, some degenerate."""
    V = rng.integers(-2, 3, (3 * n, 3)) * 0.5
    V[::7] = -0.0
    I = np.arange(3 * n).reshape(n, 3)
    I[::11, 1] = 3 * n + 5
    return V, I, rng.integers(0, 9, n)


def _spare(rng):
    """Far more vertices than corners, most of them nowhere."""
    V, I, T = _fan(9, rng)
    return np.concatenate([V, rng.random((500, 3)) * 1e6]), I, T


def _point(n, rng):
    return np.tile([[1.5, -2.0, 3.0]], (n, 1)), rng.integers(0, n, (n, 3)), np.arange(n)


CASES = {"fan16": lambda r: _fan(16, r), "fan17": lambda r: _fan(17, r), "fan2048": lambda r: _fan(2048, r),
         "fan2049": lambda r: _fan(2049, r), "book33": lambda r: _book(33, r), "book900": lambda r: _book(900, r),
         "staged": lambda r: _dense_fans(15, 300, r), "dense": lambda r: _dense_fans(16, 4000, r),
         "long": lambda r: _dense_fans(40, 300, r), "soup": lambda r: _soup(3000, r), "spare": _spare,
         "point": lambda r: _point(40, r), "points": lambda r: _point(3000, r)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_edge_lists(cuda, name):
    V, I, T = CASES[name](np.random.default_rng(len(name)))
    V, I, T = V.astype(np.float32), I.astype(np.uint32), T.astype(np.int32)
    got = api.extract_edges(torch.from_numpy(V).cuda(), torch.from_numpy(I.view(np.int32)).cuda(),
                            torch.from_numpy(T).cuda())
    want = bind.extract_edges(V, I, T)
    for g, w in zip(got, want):
        assert g.cpu().numpy().tobytes() == np.ascontiguousarray(w).tobytes()
