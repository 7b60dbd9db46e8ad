"""rs_compact_hits around its tile (4,096 points): sizes at and beside its edges, many tiles
(look-back), no hits, only hits, pointers off the 16-byte boundary, a capacity below the
count and outputs left out, and several streams and threads at once."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from rayspace3d_gb300 import _lib, api

pytestmark = pytest.mark.gpu


def _objects(n, share, seed):
    rng = np.random.default_rng(seed)
    o = np.full(n, -1, np.int32)
    k = rng.random(n) < share
    o[k] = rng.integers(-2 ** 31, 2 ** 31 - 1, k.sum())
    return o


def _compact(t, capacity, ids=True, objs=True, stream=None):
    n = t.numel()
    out = [torch.full((max(n, 1),), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
    cnt = ctypes.c_uint64(99)
    st = _lib.load().rs_compact_hits(t.data_ptr(), n, out[0].data_ptr() if ids else None,
                                     out[1].data_ptr() if objs else None, capacity, ctypes.byref(cnt),
                                     stream.cuda_stream if stream else torch.cuda.current_stream().cuda_stream)
    return st, cnt.value, out[0].cpu().numpy(), out[1].cpu().numpy()


@pytest.mark.parametrize("share", [0.0, 0.1, 1.0])
@pytest.mark.parametrize("n", [1, 3, 4, 255, 4095, 4096, 4097, 8192, 131071, 1300001])
def test_compaction(cuda, n, share):
    o = _objects(n + 1, share, n)
    for off in (0, 1):  # aligned, and one element off
        h = o[off:off + n]
        t = torch.from_numpy(o).cuda()[off:off + n]
        want = np.nonzero(h != -1)[0].astype(np.int32)
        st, c, ids, objs = _compact(t, n)
        assert st == 0 and c == len(want)
        assert np.array_equal(ids[:c], want) and np.array_equal(objs[:c], h[want])
        assert (ids[c:] == -7).all() and (objs[c:] == -7).all()
    cap = len(want) // 2
    st, c, ids, objs = _compact(t, cap, ids=share > 0.5)
    assert c == len(want) and st == (_lib.RS_ERR_OUTPUT_OVERFLOW if c > cap else 0)
    assert np.array_equal(objs[:cap], h[want[:cap]]) and (objs[cap:] == -7).all()


def test_threads_and_streams(cuda):
    """Calls in flight at once have words of their own."""
    from rayspace3d_gb300 import gen
    mesh = gen.instanced_set(300, 1, 0.5, 2.0, 12.0, seed=5)
    bvh = api.Bvh(mesh)
    pts = gen.mesh_points(mesh, 60000, seed=6)
    want = api.point_in_mesh(bvh, pts)[0].cpu().numpy()
    hits = np.nonzero(want != -1)[0]
    bad = []

    def work():
        s = torch.cuda.Stream()
        for _ in range(20):
            with torch.cuda.stream(s):
                obj, _ = api.point_in_mesh(bvh, pts, stream=s)
                ids, objs = api.compact_hits(obj, stream=s)
                s.synchronize()
                if not (np.array_equal(obj.cpu().numpy(), want) and np.array_equal(ids.cpu().numpy(), hits) and
                        np.array_equal(objs.cpu().numpy(), want[hits])):
                    bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
