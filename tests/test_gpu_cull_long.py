"""Broad phase of objects of many triangles (the lists of overlapping boxes, k_box_pairs) and
of packets of objects: no overlap, fewer and more partners than a list holds, objects that
lie inside others without touching them, and one object a side.  The pair set equals the
CPU oracle's and the join's without a broad phase."""
import numpy as np
import pytest

from oracle import bind
from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _spheres(level, centres, radii, seed):
    rng = np.random.default_rng(seed)
    n = len(centres)
    V, I, T = synth.assemble_uniform(level, np.asarray(radii, float), synth.random_rotations(rng, n),
                                     np.asarray(centres, float))
    return synth.make_geometry(V, I, T)


def _pair(level, n, world, seed, r=(0.5, 2.0)):
    rng = np.random.default_rng(seed)
    return [_spheres(level, rng.uniform(0, world, (n, 3)), rng.uniform(*r, n), seed + k) for k in (1, 2)]


def _nested(level):
    """B objects deep inside A objects, in hollows without a triangle, and some that cross."""
    rng = np.random.default_rng(4)
    c = rng.uniform(0, 30, (12, 3))
    A = _spheres(level, c, np.full(12, 5.0), 5)
    B = _spheres(level, np.concatenate([c, c[:6] + 4.9]), np.concatenate([np.full(12, 2.0), np.full(6, 1.0)]), 6)
    return A, B


CASES = {"one": lambda: _pair(4, 1, 0.5, 1, (1.0, 1.1)), "apart": lambda: _pair(3, 20, 200.0, 2), "some": lambda: _pair(3, 30, 8.0, 3),
         "many": lambda: _pair(3, 40, 4.0, 4), "nested": lambda: _nested(4), "few triangles": lambda: _pair(1, 900, 22.0, 5),
         "packets": lambda: _pair(0, 6000, 60.0, 6)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_partners(cuda, name):
    A, B = CASES[name]()
    a, b = api.Bvh(api.DeviceGeometry(A)), api.Bvh(api.DeviceGeometry(B))
    want = bind.overlap_join(A, B)
    L = _lib.load()
    for cull in (1, 0):
        L.rs_set_overlap_cull(cull)
        try:
            ps = api.PairSet(1 << 14)
            api.overlap_join(a, b, ps)
        finally:
            L.rs_set_overlap_cull(1)
        np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)
    assert name == "apart" or len(want) > 0
