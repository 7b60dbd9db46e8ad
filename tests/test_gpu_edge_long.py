"""Edges with long crossing lists and wide traversals: lists of a few and of many edges with
as many crossings as a packet keeps and one more, and, on the warp-per-edge path, 255 to 1400
crossings of one edge (512 is what a warp keeps), hundreds of crossings at one distance, and edges
of large objects through a dense cluster, whose packets run out of steps.  Pair sets equal the CPU
oracle's."""
import numpy as np
import pytest

from oracle import bind
from rayspace3d_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _rod(length):
    return synth.box_set([(np.array([0.05, 0.03, -0.5]), np.array([0.15, 0.11, length]))])


def _slabs(k):
    """k slabs across the rod: its long edges cross 2 k faces."""
    return synth.box_set([(np.array([-1.0, -1.0, 0.02 * j]), np.array([1.0, 1.0, 0.02 * j + 0.013])) for j in range(k)])


def _half(k):
    """k slabs, one of which holds the rods' ends: an odd number of crossings."""
    return synth.box_set([(np.array([-1.0, -1.0, 0.02 * j]), np.array([1.0, 1.0, 0.02 * j + 0.013]))
                          for j in range(k - 1)] + [(np.array([-1.0, -1.0, -1.0]), np.array([1.0, 1.0, -0.2]))])


def _coincident(k):
    """k equal boxes and 40 slabs behind them: 2 k crossings at two distances."""
    return synth.box_set([(np.array([-1.0, -1.0, 0.1]), np.array([1.0, 1.0, 0.3]))] * k +
                         [(np.array([-1.0, -1.0, 0.5 + 0.02 * j]), np.array([1.0, 1.0, 0.51 + 0.02 * j]))
                          for j in range(40)])


def _cluster(n):
    rng = np.random.default_rng(9)
    V, I, T = synth.assemble_uniform(1, np.full(n, 2.5), None, rng.normal(0.0, 12.0, (n, 3)))
    return synth.make_geometry(V, I, T)


def _large(n):
    rng = np.random.default_rng(10)
    V, I, T = synth.assemble_uniform(0, rng.uniform(15.0, 45.0, n), None, rng.normal(0.0, 6.0, (n, 3)))
    return synth.make_geometry(V, I, T)


def _rods(k):
    """k rods side by side through the same slabs: a list of 18 k edges of 8 or 9 crossings."""
    return synth.box_set([(np.array([0.001 * j, 0.03, -0.5]), np.array([0.001 * j + 0.0004, 0.11, 4.0]))
                          for j in range(k)])


CASES = {"8 crossings": lambda: (_rods(1), _slabs(4)), "9 crossings": lambda: (_rods(1), _half(5)),
         "594 edges": lambda: (_rods(33), _half(5)), "3600 edges": lambda: (_rods(200), _slabs(4)), "256": lambda: (_rod(4.0), _slabs(128)), "255": lambda: (_rod(4.0), _half(128)),
         "258": lambda: (_rod(4.0), _slabs(129)), "511": lambda: (_rod(6.0), _half(256)),
         "512": lambda: (_rod(6.0), _slabs(256)), "514": lambda: (_rod(6.0), _slabs(257)),
         "700": lambda: (_rod(8.0), _slabs(350)), "1400": lambda: (_rod(15.0), _slabs(700)),
         "equal": lambda: (_rod(4.0), _coincident(300)), "equal, more": lambda: (_rod(4.0), _coincident(600)),
         "large cluster": lambda: (_large(400), _cluster(40000)), "cluster": lambda: (_large(60), _cluster(6000))}


@pytest.mark.parametrize("rule", [(100, False), (100000, False), (256, True)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_long_edges(cuda, name, rule):
    A, B = CASES[name]()
    ps = api.PairSet(1 << 20)
    ps.set_edge_rule(*rule)
    bb = api.Bvh(api.DeviceGeometry(B))
    api.edge_join(bb, api.DeviceGeometry(A), ps)
    want = bind.edge_join(A.edges, B.vertices, B.indices, B.tri2obj, max_hits=rule[0], next_float=rule[1])
    assert len(want) > 0
    np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)
