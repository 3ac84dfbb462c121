"""Calls after one that ended in a CUDA error that leaves the device usable."""
import numpy as np
import pytest

from oracle import idx

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


def test_the_next_call_does_not_see_the_error(tmp_path):
    n, K, d = 16, 4, 38720  # rows wider than the verification's shared memory takes
    ids = ((np.arange(n)[:, None] + np.arange(1, K + 1)) % n).astype(np.uint32)
    adj = np.concatenate([np.full((n, 1), K, np.uint32), ids, np.zeros((n, 4), np.uint32)], 1)
    p = str(tmp_path / "wide.idx")
    X = np.random.default_rng(0).standard_normal((n, d)).astype(np.float32)
    idx.write_idx(p, X, ids, np.ones((n, K), np.float32), np.full(n, K, np.uint32), M=4, adj0=adj)
    wide = H.HRNN.load(p, d)
    wide.buildRKNNG()
    with pytest.raises(H.HrnnError, match="SharedMemory"):
        wide.search_rknn_batch(X[:3], 2, K, 8, k=3)
    again = H.HRNN.load(p, d)
    again.buildRKNNG()
    assert len(again.get_rknng()[1]) == n * K
