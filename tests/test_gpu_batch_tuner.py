"""The batch tuner times every leaf size and chunk once: the traversal stack's depth, which the
call also reports, changes no kernel; the option is checked as before and changes no result."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def test_each_configuration_is_timed_once(cuda):
    L = _lib.load()
    g, pts = synth.pim_workload(5000, level=2)
    dg = api.DeviceGeometry(g)
    bvh = api.Bvh(dg)
    p = torch.from_numpy(pts).cuda()
    obj = torch.empty(len(pts), dtype=torch.int32, device="cuda")
    inside = torch.empty(len(pts), dtype=torch.uint8, device="cuda")
    d = (0.36, -0.48, 0.8)  # no column grid
    h = ctypes.c_void_p()
    assert L.rs_batch_create(ctypes.byref(h)) == 0
    try:
        assert L.rs_batch_add_pim(h, bvh.handle, p.data_ptr(), len(pts), *d, obj.data_ptr(), inside.data_ptr(), None) == 0
        leaf, chunk, depth, ms = ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_double()
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        n0 = L.rs_launch_count()
        api.Bvh(dg).close()
        build = L.rs_launch_count() - n0
        n0 = L.rs_launch_count()
        assert L.rs_batch_autotune(h, ctypes.byref(leaf), ctypes.byref(chunk), ctypes.byref(depth), ctypes.byref(ms), s) == 0
        # Four builds and the chosen one; two launches, three times, for four leaf sizes and three chunks.
        assert L.rs_launch_count() - n0 <= 5 * (build + 4) + 2 * 3 * 12
        assert leaf.value in (2, 4, 8, 16) and chunk.value in (32, 64, 128) and depth.value == 64 and ms.value > 0
        want = bind.pim(g.vertices, g.indices, g.tri2obj, pts, direction=d)
        for option, ok in ((32, True), (64, True), (0, True), (48, False)):
            assert (L.rs_batch_set_options(h, 0, option, 1) == 0) == ok
            obj.fill_(7)
            assert L.rs_batch_submit(h, s) == 0 and L.rs_batch_wait(h, None) == 0
            np.testing.assert_array_equal(obj.cpu().numpy(), want)
            np.testing.assert_array_equal(inside.cpu().numpy().astype(bool), want >= 0)
    finally:
        L.rs_batch_destroy(h)
