"""Containment rays at the lengths where their path changes: a warp's crossing list (512) is
filled exactly, passed by one object, and far exceeded; objects whose triangles are not
stored together; one object alone.  Pair sets equal the CPU oracle's."""
import numpy as np
import pytest

from oracle import bind
from rayspace3d_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _nested(k):
    """k concentric cubes: a ray from the centre crosses each once, and contains it."""
    return synth.box_set([(np.full(3, -1.0 - 0.01 * j), np.full(3, 1.0 + 0.01 * j)) for j in range(k)], edges=True)


def _stacked(k):
    """k boxes above the origin, crossed twice each, around 3 boxes that hold it."""
    boxes = [((-1.0, -1.0, 2.0 + j), (1.0, 1.0, 2.5 + j)) for j in range(k)]
    boxes += [((-2.0, -2.0, -2.0 - j), (2.0, 2.0, 2.0 * k + 4.0 + j)) for j in range(3)]
    return synth.box_set([(np.asarray(a), np.asarray(b)) for a, b in boxes], edges=True)


def _sources(n):
    rng = np.random.default_rng(3)
    c = rng.uniform(-0.4, 0.4, (n, 3))
    return synth.box_set([(p - 0.05, p + 0.05) for p in c], edges=True)


def _keys(A, B, shuffle):
    if shuffle:  # the objects' triangles interleaved
        p = np.random.default_rng(5).permutation(len(A.indices))
        A = synth.make_geometry(A.vertices, A.indices[p], A.tri2obj[p])
    da, db = api.DeviceGeometry(A), api.DeviceGeometry(B)
    ps = api.PairSet(1 << 14)
    api.containment(api.Bvh(db), da, ps)
    got = ps.finalize().cpu().numpy().astype(np.uint64)
    want = bind.containment(A, B.vertices, B.indices, B.tri2obj)
    assert np.array_equal(np.sort(got), np.sort(want))
    join = api.PairSet(1 << 14)
    api.overlap_join(api.Bvh(da), api.Bvh(db), join, with_containment=True)
    assert np.array_equal(join.finalize().cpu().numpy().astype(np.uint64), bind.intersection_join(A, B))
    return len(want)


@pytest.mark.parametrize("target", [_nested(32), _nested(33), _nested(512), _nested(513), _stacked(254), _stacked(700)],
                         ids=["32", "33", "512", "513", "511", "1403"])
@pytest.mark.parametrize("n,shuffle", [(1, False), (70, True)])
def test_containment_lists(cuda, target, n, shuffle):
    assert _keys(_sources(n), target, shuffle) > 0
