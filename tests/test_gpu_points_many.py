"""Points whose rays cross more triangles than a query's own list holds (8 in a packet, 256 on a
column grid) up to several ranges of 512: boxes around and above the points, hundreds of
crossings at one distance, distances closer than the advance step and beyond it, all kinds of
direction, single calls, filtered calls and batches.  Objects and parities equal the CPU
oracle's, and the time stays near that of rays which the lists hold."""
import ctypes
import time

import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _nested(k, step=0.002):
    return [(np.full(3, -1.0 - step * j), np.full(3, 1.0 + step * j)) for j in range(k)]


def _stacked(k, gap=0.02):
    return [(np.array([-1.5, -1.5, 2.5 + gap * j]), np.array([1.5, 1.5, 2.5 + gap * (j + 0.5)])) for j in range(k)]


def _far(boxes):
    return [(lo + [0, 0, 40.0], hi + [0, 0, 40.0]) for lo, hi in boxes]


CASES = {"9 nested": lambda: _nested(9), "65 nested": lambda: _nested(65), "257 nested": lambda: _nested(257),
         "512 nested": lambda: _nested(512), "513 nested": lambda: _nested(513), "1601 nested": lambda: _nested(1601, 0.0005),
         "600 stacked": lambda: _nested(3) + _stacked(600, 0.001), "900 closer than the step": lambda: _nested(900, 3e-7),
         "300 at one distance": lambda: _nested(2) + [_nested(1, 0)[0]] * 300 + _nested(5),
         "600 at one distance": lambda: _nested(2) + [_nested(1, 0)[0]] * 600 + _stacked(200),
         "where steps do not move t": lambda: _nested(2) + _far(_stacked(300))}


def _mesh(boxes):
    g = synth.box_set(boxes, edges=False)
    p = np.random.default_rng(len(boxes)).permutation(len(boxes))
    return synth.make_geometry(g.vertices, g.indices, p[g.tri2obj], edges=False)


def _points(n):
    rng = np.random.default_rng(n)
    return rng.uniform(-1.4, 1.4, (n, 3)).astype(np.float32)


@pytest.mark.parametrize("name", sorted(CASES))
def test_single_and_batched(cuda, name):
    g, pts = _mesh(CASES[name]()), _points(77)
    bvh = api.Bvh(api.DeviceGeometry(g))
    p = torch.from_numpy(pts).cuda()
    directions = [(1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0), (0.36, -0.48, 0.8), (0.0, 0.0, -1.0)]
    want = [bind.pim(g.vertices, g.indices, g.tri2obj, pts, direction=d) for d in directions]
    L = _lib.load()
    h = ctypes.c_void_p()
    assert L.rs_batch_create(ctypes.byref(h)) == 0
    try:
        outs = []
        for d, w in zip(directions, want):
            obj, inside = api.point_in_mesh(bvh, p, direction=d)
            np.testing.assert_array_equal(obj.cpu().numpy(), w)
            np.testing.assert_array_equal(inside.cpu().numpy().astype(bool), w >= 0)
            o, i = torch.full_like(obj, 7), torch.full_like(inside, 7)
            assert L.rs_batch_add_pim(h, bvh.handle, p.data_ptr(), len(pts), *d, o.data_ptr(), i.data_ptr(), None) == 0
            outs.append((o, i))
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert L.rs_batch_submit(h, s) == 0 and L.rs_batch_wait(h, None) == 0
        for (o, i), w in zip(outs, want):
            np.testing.assert_array_equal(o.cpu().numpy(), w)
            np.testing.assert_array_equal(i.cpu().numpy().astype(bool), w >= 0)
    finally:
        L.rs_batch_destroy(h)
    obj, _ = api.point_in_mesh(bvh, p, filtered=True)
    np.testing.assert_array_equal(obj.cpu().numpy(), bind.pim(g.vertices, g.indices, g.tri2obj, pts, filtered=True))


def test_the_next_list_costs_no_traversal_a_crossing(cuda):
    p = torch.from_numpy(_points(20000)).cuda()

    def seconds(k):
        bvh = api.Bvh(api.DeviceGeometry(_mesh(_stacked(k))))
        best = np.inf
        for _ in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            api.point_in_mesh(bvh, p)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best
    assert seconds(200) < 20 * seconds(100)  # 400 crossings a ray and 200; hundreds of times, a traversal each
