"""Searches and builds with NaN and infinite distances: the team of warps and the single
warp agree, and the other queries of a batch keep their answers."""
import numpy as np
import pytest

from oracle import data

import hrnn_b200 as H

pytestmark = pytest.mark.gpu

DIMS = [64, 32, 20, 50]  # a width with its own kernel, other multiples of 16, of 4, the rest


@pytest.mark.parametrize("d", DIMS)
def test_searches_with_nan_and_huge_queries(monkeypatch, d):
    X = data.mixture(900, d, 12, 1.0, 3, 3)
    h = H.HRNN(d, 900, 8, 60, 100, 24)
    h.add_points(X)
    h.refineKNNG(2, 20)
    h.buildRKNNG()
    Q = data.mixture(9, d, 12, 1.0, 3, 77)
    monkeypatch.setenv("HRNN_TEAM", "0")
    want = h.search_rknn_batch(Q, 5, 24, 200)
    B = Q.copy()
    B[1, 0] = np.nan
    B[4] = np.nan
    B[6, d - 1] = np.inf
    B[7] = 1e30
    expanded = []
    for team in ("0", "4"):
        monkeypatch.setenv("HRNN_TEAM", team)
        got = h.search_rknn_batch(B, 5, 24, 200)
        assert all(len(got[i]) == 0 for i in (1, 4, 6, 7))
        assert all(np.array_equal(got[i], want[i]) for i in (0, 2, 3, 5, 8))
        expanded.append(h.last_search_stats()["n_expanded"])
    assert expanded[0] == expanded[1]


@pytest.mark.parametrize("d", DIMS)
@pytest.mark.parametrize("what", ["some", "all"])
def test_builds_with_nan_and_huge_points(tmp_path, monkeypatch, d, what):
    n = 700
    X = data.mixture(n, d, 12, 1.0, 5, 5)
    if what == "all":
        X[:] = np.nan
    else:
        X[5::40, 0] = np.nan
        X[9::60] = 1e30
    raw = []
    for team in ("0", "4"):
        monkeypatch.setenv("HRNN_TEAM", team)
        h = H.HRNN(d, n, 8, 60, 100, 16)
        h.add_points(X)
        p = tmp_path / f"{team}.idx"
        h.saveIndex(str(p))
        raw.append(p.read_bytes())
    assert raw[0] == raw[1]


@pytest.mark.parametrize("prec", [H.PREC_BF16, H.PREC_INT8])
@pytest.mark.parametrize("nq", [9, 900])  # one warp per block; four
def test_reduced_precision_searches_with_nan_and_huge_queries(prec, nq):
    d = 128
    h = H.HRNN(d, 3000, 16, 60, 100, 24)
    h.add_points(data.mixture(3000, d, 12, 1.0, 3, 3))
    h.refineKNNG(2, 20)
    h.buildRKNNG()
    h.set_precision(prec)
    Q = data.mixture(nq, d, 12, 1.0, 3, 77)
    want = h.search_rknn_batch(Q, 5, 24, 200)
    B = Q.copy()
    B[1, 0] = np.nan
    B[4] = np.nan
    B[6, d - 1] = np.inf
    B[7] = 1e30
    got = h.search_rknn_batch(B, 5, 24, 200)
    assert all(len(got[i]) == 0 for i in (1, 4, 6, 7))
    assert all(np.array_equal(got[i], want[i]) for i in range(nq) if i not in (1, 4, 6, 7))
