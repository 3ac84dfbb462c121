"""NNDescent local join at widths that are multiples of 4 but not of 16 (and at a
neighbouring one of each other kind): lists against the one-thread oracle."""
import numpy as np
import pytest

from oracle import data, port

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [4, 12, 20, 36, 100, 132, 200, 112, 30])
@pytest.mark.parametrize("sample", [3, 40])
def test_refined_lists_match_oracle(d, sample):
    n, K = 500, 24
    X = data.mixture(n, d, 6, 1.0, 13, 13)
    h = H.HRNN(d, n, 8, 40, 100, K)
    h.add_points(X)
    ids, dist, cnt = (np.ascontiguousarray(a).copy() for a in h.get_knng())
    new = (np.arange(K)[None, :] < cnt[:, None]).astype(np.uint8)
    lanes, fused = H.detect_l2_order()
    h.set_l2_order(lanes, fused)
    port.refine(np.ascontiguousarray(X), ids, dist, cnt, new, 3, sample, lanes, fused)
    h.refineKNNG(3, sample)
    gi, gd, gc = h.get_knng()
    assert np.array_equal(gc, cnt)
    m = np.arange(K)[None, :] < cnt[:, None]
    assert np.array_equal(gd[m], dist[m])
    # equal distances (in 4 dims) may stand in either order
    tie = (dist[:, 1:] == dist[:, :-1]) & m[:, 1:]
    rows = ~tie.any(1)
    assert rows.mean() > 0.9 and np.array_equal(gi[rows][m[rows]], ids[rows][m[rows]])
