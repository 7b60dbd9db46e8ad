"""A batch replayed on an edge payload that was rewritten in place: a replay that spills its table
leaves nothing behind in the overflow table, whether the submits before it spilled or not."""
import ctypes

import numpy as np
import pytest
import torch

from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu
BOXES, EDGES = 50, 2000


def test_replays_that_spill(cuda):
    L = _lib.load()
    c = np.zeros((BOXES, 3))
    c[:, 0] = 2.0 * np.arange(BOXES)
    target = api.Bvh(api.DeviceGeometry(synth.box_set([(p - 0.5, p + 0.5) for p in c], edges=True)))
    # Edge e crosses box e % BOXES, or lies away from all.
    at = torch.from_numpy(c[np.arange(EDGES) % BOXES] + [0.1, 0.2, 0.0]).float().cuda()
    up = torch.tensor([0.0, 0.0, 3.0], device="cuda")
    ids = torch.arange(EDGES, dtype=torch.int32, device="cuda")
    payload = [torch.zeros((EDGES, 3), device="cuda"), torch.zeros((EDGES, 3), device="cuda"), ids.clone(),
               torch.ones(EDGES, dtype=torch.int32, device="cuda"), ids.clone()]

    def rewrite(hits, first_source):
        away = (torch.arange(EDGES, device="cuda") >= hits)[:, None] * 1000.0
        payload[0].copy_(at - up + away)
        payload[1].copy_(at + up + away)
        payload[4].copy_(ids + first_source)
        return np.sort((np.arange(hits, dtype=np.uint64) + np.uint64(first_source)) << np.uint64(32)
                       | np.arange(hits, dtype=np.uint64) % np.uint64(BOXES))

    ps = api.PairSet(4)
    h = ctypes.c_void_p()
    assert L.rs_batch_create(ctypes.byref(h)) == 0
    try:
        assert L.rs_batch_add_edges(h, target.handle, *[t.data_ptr() for t in payload], EDGES, 0, ps.handle, None) == 0
        s = torch.cuda.Stream()  # a stream that can be captured
        caps = []
        for hits, first_source in ((0, 0), (40, 10000), (EDGES, 20000), (40, 10000)):
            want = rewrite(hits, first_source)
            torch.cuda.synchronize()
            ps.clear()
            assert L.rs_batch_submit(h, ctypes.c_void_p(s.cuda_stream)) == 0
            assert L.rs_batch_wait(h, None) == 0
            np.testing.assert_array_equal(ps.finalize().cpu().numpy().astype(np.uint64), want)
            caps.append(ps.info()[0])
        assert caps[0] == 4 < caps[1] < EDGES < caps[2] == caps[3]
    finally:
        L.rs_batch_destroy(h)
