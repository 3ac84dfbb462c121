"""Reduced-precision beam search at each way of reading rows: the small-batch shape
(all rows of a step in flight) against the large-batch one, and against the exact
form's answers."""
import numpy as np
import pytest

from oracle import data

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [48, 96, 128, 256])
@pytest.mark.parametrize("prec", [H.PREC_BF16, H.PREC_INT8])
def test_shapes_agree_and_find_the_exact_answers(d, prec):
    n, k = 6000, 10
    X = data.mixture(n, d, 24, 1.0, 41, 41)
    Q = data.mixture(700, d, 24, 1.0, 41, 42)
    h = H.HRNN(d, n, 16, 100, 100, 32)
    h.add_points(X)
    h.refineKNNG(4, 30)
    h.buildRKNNG()
    h.set_autotune(False)
    exact = h.search_rknn_batch(Q, 10, 32, 100, k=k)
    h.set_precision(prec)
    for m, ef in ((1, 1), (5, 33), (10, 100)):
        whole = h.search_rknn_batch(Q, m, 32, ef, k=k)
        parts = [a for i in range(0, 700, 100) for a in h.search_rknn_batch(Q[i:i + 100], m, 32, ef, k=k)]
        assert all(np.array_equal(a, b) for a, b in zip(whole, parts)), (m, ef)
    # the same proxies but for ties of near-equal distances: answers that differ are few
    same = np.mean([np.array_equal(a, b) for a, b in zip(whole, exact)])
    assert same > 0.9, same
