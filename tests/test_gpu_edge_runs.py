"""Unique edges where many records meet: one edge shared by more than a thousand objects (again
by some of them), coincident copies of a mesh, fans around one vertex below and beyond a
block's list, everything at one point.  Byte-equal to the CPU restatement; a long run of
objects takes no longer than a few times as many triangles that share nothing."""
import time

import numpy as np
import pytest
import torch

from rayspace3d_gb300 import api, gen, synth

pytestmark = pytest.mark.gpu


def _book(n, again):
    """n triangles on one edge, their objects in a mixed order, `again` of them twice."""
    rng = np.random.default_rng(n)
    V = np.concatenate([[[0, 0, 0], [1, 0, 0]], rng.uniform(1, 2, (n + again, 3))])
    i = np.arange(n + again)
    T = np.concatenate([rng.permutation(n), rng.permutation(n)[:again]])
    I = np.stack([0 * i, 0 * i + 1, i + 2], 1)
    flip = rng.random(len(I)) < 0.5
    I[flip] = I[flip][:, [1, 0, 2]]
    return V, I, T


def _copies(objects, times, level):
    g = synth.sphere_set(objects, level, 0.5, 2.0, 10.0, np.random.default_rng(times), edges=False)
    V = np.tile(g.vertices, (times, 1))
    I = np.concatenate([g.indices.astype(np.int64) + k * len(g.vertices) for k in range(times)])
    T = np.concatenate([g.tri2obj + k * objects for k in range(times)])
    p = np.random.default_rng(7).permutation(len(I))
    return V, I[p], T[p]


def _fan(n, others):
    """n triangles around one vertex, beside small spheres; a few triangles are skipped."""
    a = np.arange(n) * (2 * np.pi / n)
    rim = np.stack([np.cos(a), np.sin(a), 0 * a], 1) * 50
    g = synth.sphere_set(max(others, 1), 1, 0.5, 2.0, 100.0, np.random.default_rng(n), edges=False)
    i = np.arange(n)
    I = np.concatenate([g.indices.astype(np.int64), len(g.vertices) + np.stack([0 * i, 1 + i, 1 + (i + 1) % n], 1)])
    V = np.concatenate([g.vertices, np.zeros((1, 3)), rim])
    I[5::301, 1] = len(V) + 3
    T = np.concatenate([g.tri2obj, g.tri2obj.max() + 1 + (i % 3)])
    return V, I, T


def _point(n):
    rng = np.random.default_rng(n)
    return rng.uniform(-4e-6, 4e-6, (n, 3)), rng.integers(0, n, (n, 3)), rng.integers(0, 40, n)


CASES = {"book of 33": lambda: _book(33, 5), "book of 1300": lambda: _book(1300, 200), "book of 2048": lambda: _book(2000, 48),
         "book of 2049": lambda: _book(2049, 0), "64 copies": lambda: _copies(3, 64, 2), "600 copies": lambda: _copies(2, 600, 1),
         "900 copies": lambda: _copies(2, 900, 1), "fan of 2000": lambda: _fan(2000, 50), "fan of 6000": lambda: _fan(6000, 50),
         "one point": lambda: _point(5000), "one point, few": lambda: _point(60)}


def _device(V, I, T):
    return [torch.from_numpy(np.ascontiguousarray(a, d)).cuda() for a, d in ((V, np.float32), (I, np.int32), (T, np.int32))]


@pytest.mark.parametrize("name", sorted(CASES))
def test_payload(cuda, name):
    V, I, T = CASES[name]()
    w = synth.extract_edges(np.asarray(V, np.float32), np.asarray(I, np.uint32), np.asarray(T, np.int32))
    got = api.extract_edges(*_device(V, I, T))
    for a, b in zip(got, (w.starts, w.ends, w.offsets, w.counts, w.sources)):
        np.testing.assert_array_equal(a.cpu().numpy().view(np.uint32), np.ascontiguousarray(b).reshape(a.shape).view(np.uint32))


def _seconds(mesh):
    """Of the fastest of four extractions; mesh: host arrays or device tensors."""
    mesh = mesh if torch.is_tensor(mesh[0]) else _device(*mesh)
    best = np.inf
    for _ in range(4):
        torch.cuda.synchronize()
        t = time.perf_counter()
        api.extract_edges(*mesh)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def test_a_long_run_is_not_quadratic(cuda):
    rng = np.random.default_rng(1)
    loose = rng.uniform(0, 100, (6000, 3)), np.arange(6000).reshape(-1, 3), np.arange(2000)
    assert _seconds(_book(2000, 0)) < 20 * _seconds(loose)  # 80 times and more, looking back through the run


def test_one_long_list_does_not_start_over(cuda):
    """A vertex of more triangles than a block's list holds, beside 3.2 M others."""
    many = gen.instanced_set(10000, 2, 0.5, 2.0, 1000.0, seed=3)

    def beside(n):
        V, I, T = _device(*_fan(n, 1))
        return torch.cat([many.V, V]), torch.cat([many.I, I + many.nV]), torch.cat([many.T, T + 10000])
    assert _seconds(beside(6000)) < 3 * _seconds(beside(2000))  # 5.5 times, starting over by wide words


def test_records_of_one_rank_do_not_queue(cuda):
    """A mesh collapsed to a point, against one of as many triangles that is not."""
    V, I, T = _copies(1500, 1, 3)
    assert _seconds((V * 1e-9, I, T)) < 3 * _seconds((V, I, T))  # 5 times, with an atomic each
