"""Inserting a point needs work space for its own links, not for every list's."""
import numpy as np
import pytest

from oracle import data

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


def test_insert_into_a_large_index_on_a_nearly_full_device():
    import torch
    cap = 8_000_000
    X = data.mixture(301, 4, 4, 1.0, 1, 1)
    h = H.HRNN(4, cap, 2, 32, 100, 1)
    h.add_points(X[:300])
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - 20 * cap, dtype=torch.uint8, device="cuda")  # 20 bytes a list left
    try:
        h.add_points(X[300:])
    finally:
        del held
        torch.cuda.empty_cache()
    small = H.HRNN(4, 301, 2, 32, 100, 1)  # the same insertions without the pressure
    small.add_points(X[:300])
    small.add_points(X[300:])
    assert all(np.array_equal(a[:301], b) for a, b in zip(h.get_knng(), small.get_knng()))
