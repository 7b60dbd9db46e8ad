"""rs_pairset_finalize at the lengths where its path changes (one block's 4,096 keys, tiles
merged by rank up to 65,536, the radix sort beyond), both orders, and tables used on another
stream than the one they were created on while that one is busy."""
import ctypes

import numpy as np
import pytest
import torch

from rayspace3d_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _source(n):
    """n edges from object i mod 997 + 3 i, all through one box: n distinct pairs."""
    e = np.zeros((n, 3), np.float32)
    e[:, 0] = -1.0
    f = e.copy()
    f[:, 0] = 1.0
    ids = (np.arange(n, dtype=np.int64) * 7919 % (4 * n + 1)).astype(np.int32)
    ar = np.arange(n, dtype=np.int32)
    t = [torch.from_numpy(x).cuda() for x in (e, f, ar, np.ones(n, np.int32), ids)]
    V = torch.zeros((3, 3), device="cuda")
    return api.DeviceGeometry.from_tensors(V, torch.tensor([[0, 1, 2]], dtype=torch.int32, device="cuda"),
                                           torch.zeros(1, dtype=torch.int32, device="cuda"), edges=t), ids


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 8192, 9072, 65535, 65536, 65537])
def test_sorted_keys(cuda, n):
    box = synth.box_set([(np.full(3, -0.5), np.full(3, 0.5))])
    bvh = api.Bvh(api.DeviceGeometry(box))
    src, ids = _source(n)
    ids = np.unique(ids).astype(np.uint64)
    for swap in (False, True):
        ps = api.PairSet(1 << 10)
        api.edge_join(bvh, src, ps, swap=swap)
        for order in (0, 1):
            got = ps.finalize(order=order).cpu().numpy().astype(np.uint64)
            want = ids if swap else ids << np.uint64(32)
            assert np.array_equal(got, want)
    if n > 4096:  # a result buffer one short
        out = torch.full((len(ids),), -1, dtype=torch.int64, device="cuda")
        c = ctypes.c_uint64()
        st = _lib.load().rs_pairset_finalize(ps.handle, 0, out.data_ptr(), len(ids) - 1, ctypes.byref(c),
                                             torch.cuda.current_stream().cuda_stream)
        assert st == _lib.RS_ERR_OUTPUT_OVERFLOW and c.value == len(ids)


def test_created_on_a_busy_stream(cuda):
    """A new table is empty to every stream, however late its creation stream clears it."""
    box = synth.box_set([(np.full(3, -0.5), np.full(3, 0.5))])
    bvh = api.Bvh(api.DeviceGeometry(box))
    src, ids = _source(3000)
    want = np.unique(ids).astype(np.uint64) << np.uint64(32)
    junk = torch.randint(0, 1 << 40, (1 << 22,), device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for rep in range(6):
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            for _ in range(20):
                torch.sort(junk)
        ps = api.PairSet(1 << 14, stream=a)
        if rep % 3 == 1:
            ps.clear(stream=b)
        if rep % 3 == 2:
            assert ps.info(stream=b)[1] == 0 and ps.finalize(stream=b).numel() == 0
        api.edge_join(bvh, src, ps, stream=b)
        got = ps.finalize(stream=b)
        b.synchronize()
        assert np.array_equal(got.cpu().numpy().astype(np.uint64), want)
        ps.close()
