"""The widest rows the exact verification's shared memory takes: answers against the
oracle."""
import numpy as np
import pytest

from oracle import idx, port

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


# the last multiples of 16 where query, table and lists fit in 227 KB, without and with
# the counters of a threshold above 1
@pytest.mark.parametrize("d,threshold", [(38688, 1.0), (32128, 2.0)])
def test_widest_rows(tmp_path, d, threshold):
    n, K = 40, 8
    r = np.random.default_rng(d)
    X = r.standard_normal((n, d)).astype(np.float32)
    lanes, fused = H.detect_l2_order()
    D = np.stack([port.l2_batch(np.repeat(X[i:i + 1], n, 0), X, lanes, fused) for i in range(n)])
    np.fill_diagonal(D, np.inf)
    ids = np.argsort(D, 1)[:, :K].astype(np.uint32)
    dist = np.take_along_axis(D, ids.astype(np.int64), 1).astype(np.float32)
    adj = np.concatenate([np.full((n, 1), K, np.uint32), ids], 1)
    p = str(tmp_path / "wide.idx")
    idx.write_idx(p, X, ids, dist, np.full(n, K, np.uint32), M=4, adj0=adj)
    h = H.HRNN.load(p, d, device=0)
    h.buildRKNNG()
    p2 = str(tmp_path / "built.idx")
    h.saveIndex(p2)
    Q = (X[:6] + 0.5 * r.standard_normal((6, d))).astype(np.float32)
    want = port.OracleIndex(idx.read_idx(p2)).search_batch(Q, 4, K, 20, threshold=threshold, k=5)
    got = h.search_rknn_batch(Q, 4, K, 20, threshold=threshold, k=5)
    assert sum(map(len, want)) > 0
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
