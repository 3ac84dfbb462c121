"""BF16 form with link rows of more than 33 words (M above 16), which the two-parent
search does not take: answers against the exact form's."""
import numpy as np
import pytest

from oracle import data

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [96, 128, 256])
def test_answers_of_the_reference_order_search(d):
    X = data.mixture(6000, d, 24, 1.0, 41, 41)
    Q = data.mixture(300, d, 24, 1.0, 41, 42)
    h = H.HRNN(d, 6000, 24, 100, 100, 32)
    h.add_points(X)
    h.refineKNNG(4, 30)
    h.buildRKNNG()
    exact = h.search_rknn_batch(Q, 10, 32, 100, k=10)
    h.set_precision(H.PREC_BF16)
    got = h.search_rknn_batch(Q, 10, 32, 100, k=10)
    # the same proxies but for ties of near-equal distances: answers that differ are few
    assert np.mean([np.array_equal(a, b) for a, b in zip(got, exact)]) > 0.9
