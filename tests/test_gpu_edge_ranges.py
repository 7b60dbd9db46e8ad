"""Edges of more crossings than a warp's list holds (512), in several ranges of t: boxes around each
other, closer than the advance step, and hundreds of faces at one distance, with few and many
hits taken an edge.  Pair sets equal the CPU oracle's, and the time stays near the crossings'."""
import time

import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _nested(k, step):
    return [(np.full(3, -1.0 - step * j), np.full(3, 1.0 + step * j)) for j in range(k)]


def _target(boxes):
    g = synth.box_set(boxes, edges=False)
    p = np.random.default_rng(len(boxes)).permutation(len(boxes))
    return synth.make_geometry(g.vertices, g.indices, p[g.tri2obj])


def _sources(n, length):
    c = np.random.default_rng(n).uniform(-0.4, 0.4, (n, 3))
    return synth.box_set([(p - 0.01, p + [0.01, 0.02, length]) for p in c])


CASES = {"500": lambda: _nested(500, 0.002), "520": lambda: _nested(520, 0.002), "1100": lambda: _nested(1100, 0.001),
         "2100": lambda: _nested(2100, 0.0005), "900 closer than the step": lambda: _nested(900, 3e-7),
         "600 at one distance": lambda: _nested(3, 0.01) + [_nested(1, 0)[0]] * 600 + _nested(20, 0.02)}


@pytest.mark.parametrize("rule", [(100, False), (5000, False), (5000, True)], ids=["100", "all", "next float"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_pairs(cuda, name, rule):
    A, B = _sources(12, 3.0), _target(CASES[name]())
    ps = api.PairSet(1 << 16)
    ps.set_edge_rule(*rule)
    api.edge_join(api.Bvh(api.DeviceGeometry(B)), api.DeviceGeometry(A), ps)
    want = bind.edge_join(A.edges, B.vertices, B.indices, B.tri2obj, max_hits=rule[0], next_float=rule[1])
    np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)


def test_a_full_list_does_not_start_over(cuda):
    src = api.DeviceGeometry(_sources(8000, 2.5 + 2.0))

    def seconds(k):
        b = api.Bvh(api.DeviceGeometry(_target(_nested(k, 0.001))))
        ps, best = api.PairSet(1 << 22), np.inf
        for _ in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            api.edge_join(b, src, ps)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best
    a, b = seconds(60), seconds(2000)
    print(f"60 boxes {a * 1e3:.2f} ms, 2000 {b * 1e3:.2f} ms, {b / a:.1f} times")
    assert b < 23 * a
