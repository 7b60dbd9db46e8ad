"""Column grids of long, flat and endless scenes, whose cells are not square: strips across a band
100,000 times as long as it is wide, a wall that projects to a line, a triangle with a corner at
infinity.  Objects equal those of the traversal without a grid in all three directions, and the
CPU oracle's where every coordinate is finite, as its integers need."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _scene(kind):
    rng = np.random.default_rng(7)
    if kind == "wall":  # in the plane x = 1
        lo = np.stack([np.ones(3000), rng.uniform(0, 1, 3000), np.arange(3000) * 0.01], 1)
        boxes = [(p, p + [0.0, 5.0, 0.008]) for p in lo]
    else:
        lo = np.stack([np.sort(rng.uniform(0, 1e5, 6000)), np.zeros(6000), rng.uniform(0, 1, 6000)], 1)
        boxes = [(p, p + [3.0, 1.0, 0.5]) for p in lo]
    g = synth.box_set(boxes, edges=False)
    if kind == "endless":
        V, I = np.concatenate([g.vertices, [[np.inf, 0, 0]]]), g.indices.copy()
        I[5, 0] = len(V) - 1
        g = synth.make_geometry(V, I, g.tri2obj, edges=False)
    at = rng.integers(0, len(boxes), 3000)
    pts = np.array([boxes[k][0] for k in at]) + rng.uniform(-0.4, 1.2, (3000, 3)) * np.array([3.0, 1.0, 0.5])
    return g, pts.astype(np.float32)


@pytest.mark.parametrize("kind", ["band", "wall", "endless"])
def test_objects(cuda, kind):
    g, pts = _scene(kind)
    dg = api.DeviceGeometry(g)
    bvh, no_grid = api.Bvh(dg), api.Bvh(dg)
    p = torch.from_numpy(pts).cuda()
    inside = torch.empty(len(pts), dtype=torch.uint8, device="cuda")
    for d in ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0)):
        obj, _ = api.point_in_mesh(bvh, p, direction=d)
        want = torch.empty_like(obj)  # this entry point never builds a grid
        assert _lib.load().rs_pim_noalloc(no_grid.handle, p.data_ptr(), len(pts), *d, want.data_ptr(), inside.data_ptr(), 0,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        np.testing.assert_array_equal(obj.cpu().numpy(), want.cpu().numpy())
        if kind != "endless":
            np.testing.assert_array_equal(obj.cpu().numpy(), bind.pim(g.vertices, g.indices, g.tri2obj, pts, direction=d))
