"""The closed form of the filter-refine's box parity (rs_pim.cu, box_filter) against the
oracle's 12 exact triangle tests: points on faces, edges and corners, one float inside and
outside, far away (where t + 1e-6 rounds to t) and flat boxes, all three axes."""
import numpy as np
import pytest

from oracle import bind


def closed_form(lo, hi, pts, axis):
    """Parity of a +e_axis ray against the box, as box_filter computes it."""
    u, v = (axis + 1) % 3, (axis + 2) % 3
    inside = (pts[:, u] >= lo[u]) & (pts[:, u] < hi[u]) & (pts[:, v] >= lo[v]) & (pts[:, v] < hi[v])
    odd = np.zeros(len(pts), bool)
    for i in np.nonzero(inside)[0]:
        thr, count = np.float32(1e-6), 0
        for end in (lo[axis], hi[axis]):
            t = np.float32(end - pts[i, axis])
            if np.float32(1e-6) <= t <= np.float32(1e16) and count < 10000 and t >= thr and t < np.float32(1e16):
                count += 1
                nxt = np.float32(t + np.float32(1e-6))
                if not nxt > t:
                    count = 10000
                thr = nxt
        odd[i] = count & 1
    return odd


@pytest.mark.parametrize("seed", range(6))
def test_closed_form_equals_triangle_parity(seed):
    rng = np.random.default_rng(seed)
    lo = rng.choice([0.0, -1.0, 0.5, 3.25, -40.0], 3).astype(np.float32)
    hi = (lo + rng.choice([0.0 if seed == 0 else 0.5, 1.0, 0.25, 33.0, 100.0], 3)).astype(np.float32)
    V, F = bind.box_mesh(np.stack([lo, hi]))
    ticks = [np.concatenate([[a, b, a - 1, b + 1, (a + b) / 2, np.nextafter(b, np.float32(-1e9)),
                              np.nextafter(a, np.float32(-1e9))], rng.uniform(a - 50, b + 5, 3)])
             for a, b in zip(lo, hi)]
    pts = np.array(np.meshgrid(*ticks)).reshape(3, -1).T.astype(np.float32)
    for axis in range(3):
        d = [0.0, 0.0, 0.0]
        d[axis] = 1.0
        want = bind.pim(V, F, np.zeros(len(F), np.int32), pts, direction=tuple(d)) >= 0
        assert np.array_equal(closed_form(lo, hi, pts, axis), want)
