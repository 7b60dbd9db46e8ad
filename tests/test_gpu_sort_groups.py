"""Radix sort passes whose tiles (3,072 keys) are summed in groups of 16 for the look-back:
one key less and more than whole groups, a few tiles, and more tiles than run at once.  The
vertices of a soup of distinct positions are sorted on the way to its unique edges
(rs_extract_edges), whose payload equals the oracle's byte for byte."""
import numpy as np
import pytest
import torch

from oracle import bind
from rayspace3d_gb300 import api

pytestmark = pytest.mark.gpu
TILE = 3072


@pytest.mark.parametrize("corners", [2 * TILE + 3, 15 * TILE, 16 * TILE, 16 * TILE + 3, 32 * TILE, 33 * TILE + 3,
                                     700 * TILE + 3])
def test_sort_groups(cuda, corners):
    rng = np.random.default_rng(corners)
    n = corners // 3
    V = (rng.random((n, 1, 3)) * 100 + rng.random((n, 3, 3))).reshape(-1, 3).astype(np.float32)
    I = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    T = np.arange(n, dtype=np.int32)
    got = api.extract_edges(torch.from_numpy(V).cuda(), torch.from_numpy(I.view(np.int32)).cuda(),
                            torch.from_numpy(T).cuda())
    want = bind.extract_edges(V, I, T)
    for g, w in zip(got, want):
        assert g.cpu().numpy().tobytes() == np.ascontiguousarray(w).tobytes()
