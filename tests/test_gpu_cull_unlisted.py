"""Broad phase of objects of many triangles (k_box_pairs) against triangles that no object's box
holds: ids below zero, alone near an object or beside listed partners, and triangles without a
number in one coordinate, whose object has other triangles.  The pair set is the join's without
a broad phase, and has the pairs of those triangles."""
import numpy as np
import pytest

from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu
LEVEL = 4  # 5,120 triangles an object: the lists are used


def _spheres(centres, radii):
    n = len(centres)
    V, I, T = synth.assemble_uniform(LEVEL, np.asarray(radii, float), synth.random_rotations(np.random.default_rng(n), n),
                                     np.asarray(centres, float))
    return V, I, T


def _geometry(V, I, T, edges_of=None):
    g = synth.make_geometry(V, I, T, edges=False)
    g.edges = synth.extract_edges(V, I if edges_of is None else edges_of, T)
    return api.DeviceGeometry(g)


def _pairs(a, b, cull, swap, one_way=False):
    """(object of a, object of b); one_way: by a's edges alone."""
    L = _lib.load()
    L.rs_set_overlap_cull(cull)
    try:
        ps = api.PairSet(1 << 12)
        if swap:
            api.overlap_join(b, a, ps, direction=2 if one_way else 0)
        else:
            api.overlap_join(a, b, ps, direction=1 if one_way else 0)
    finally:
        L.rs_set_overlap_cull(1)
    p = {tuple(x) for x in api.keys_to_pairs(ps.finalize()).tolist()}
    return {(j, i) for i, j in p} if swap else p


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("beside", [False, True])
def test_ids_below_zero(cuda, beside, swap):
    """A's object 0 crosses a sphere of id -1, and (beside) one of id 0 too; object 1 crosses a sphere of id 1."""
    V, I, T = _spheres([(0, 0, 0), (100, 0, 0)], [5.0, 5.0])
    a = api.Bvh(_geometry(V, I, T))
    V, I, T = _spheres([(5, 0, 0), (0, 5, 0) if beside else (0, 50, 0), (100, 5, 0)], [1.0, 1.0, 1.0])
    T = T - 1
    T[T == 1] = 2  # an id between without triangles
    b = api.Bvh(_geometry(V, I, T))
    for one_way in (True, False):  # edges of an id below zero are always traced
        got = _pairs(a, b, 1, swap, one_way)
        assert got == _pairs(a, b, 0, swap, one_way)
        assert got == ({(0, -1), (1, 2)} | ({(0, 0)} if beside else set()))


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_triangle_without_a_number(cuda, axis, swap):
    """Sphere 0 of B has one triangle whose corners have no coordinate on an axis; A's object 0
    crosses spheres 0 and 1, object 1 crosses sphere 2, and A's objects have such a triangle too."""
    def side(centres, radii):
        V, I, T = _spheres(centres, radii)
        hurt = np.zeros((3, 3), np.float32)
        hurt[:, axis] = np.nan
        I2 = I.copy()
        I2[7] = np.arange(len(V), len(V) + 3)
        V = np.concatenate([V, hurt])
        return api.Bvh(_geometry(V, I2, T, edges_of=I))
    a = side([(0, 0, 0), (100, 0, 0), (200, 0, 0)], [5.0, 5.0, 5.0])
    b = side([(5, 0, 0), (0, 5, 0), (100, 5, 0)], [1.0, 1.0, 1.0])
    got = _pairs(a, b, 1, swap)
    assert got == {(0, 0), (0, 1), (1, 2)} == _pairs(a, b, 0, swap)
