"""Exact beam search and construction at every way of reading rows, one warp per
query / point and a team of warps (small batches): answers and expansion counts
against the oracle, graphs against each other and against a sequential insertion."""
import numpy as np
import pytest

from oracle import data, idx, port

import hrnn_b200 as H

pytestmark = pytest.mark.gpu

# unrolled widths, other multiples of 16, multiples of 4, the general path
DIMS = [64, 96, 128, 256, 32, 272, 20, 100, 260, 50]


def _build(d, n, M=8, efc=60, K=24, seed=3):
    X = data.mixture(n, d, 12, 1.0, seed, seed)
    h = H.HRNN(d, n, M, efc, 100, K)
    h.add_points(X)
    h.refineKNNG(2, 20)
    h.buildRKNNG()
    return X, h


@pytest.mark.parametrize("d", DIMS)
def test_team_and_single_warp_searches_match_oracle(tmp_path, monkeypatch, d):
    X, h = _build(d, 900)
    p = str(tmp_path / "t.idx")
    h.saveIndex(p)
    O = port.OracleIndex(idx.read_idx(p))
    Q = data.mixture(41, d, 12, 1.0, 3, 77)
    # beams of one entry, across the register beams' sizes (256, 512), and one that
    # visits more ids than the team's exact set holds
    for m, ef in ((1, 1), (3, 33), (5, 200), (5, 256), (5, 300), (5, 512), (5, 700)):
        want = O.search_batch(Q, m, 24, ef)
        exp = sum(O.search_one(q, m, 24, ef)[2]["n_expanded"] for q in Q)
        for team in ("0", "4"):
            monkeypatch.setenv("HRNN_TEAM", team)
            got = h.search_rknn_batch(Q, m, 24, ef)
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), (m, ef, team)
            assert h.last_search_stats()["n_expanded"] == exp, (m, ef, team)


def test_team_search_beyond_the_visited_set(tmp_path, monkeypatch):
    """More ids visited than the team's exact set takes (three quarters of 8192): one
    Gaussian, where neighbourhoods overlap little."""
    X = data.mixture(30000, 32, 1, 1.0, 3, 3)
    h = H.HRNN(32, 30000, 16, 60, 100, 10)
    h.add_points(X)
    h.refineKNNG(1, 10)
    h.buildRKNNG()
    p = str(tmp_path / "t.idx")
    h.saveIndex(p)
    O = port.OracleIndex(idx.read_idx(p))
    Q = data.mixture(12, 32, 1, 1.0, 3, 78)
    want = O.search_batch(Q, 5, 10, 512)
    stats = [O.search_one(q, 5, 10, 512)[2] for q in Q]
    assert max(s["n_dist"] for s in stats) > 6144
    monkeypatch.setenv("HRNN_TEAM", "4")
    got = h.search_rknn_batch(Q, 5, 10, 512)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert h.last_search_stats()["n_expanded"] == sum(s["n_expanded"] for s in stats)


@pytest.mark.parametrize("d", DIMS)
@pytest.mark.parametrize("efc", [40, 300])
def test_team_and_single_warp_builds_make_the_same_graph(tmp_path, monkeypatch, d, efc):
    raw = []
    for team in ("0", "4"):
        monkeypatch.setenv("HRNN_TEAM", team)
        X = data.mixture(1500, d, 12, 1.0, 5, 5)
        h = H.HRNN(d, 1500, 8, efc, 100, 16)
        h.add_points(X)
        p = tmp_path / f"{team}.idx"
        h.saveIndex(str(p))
        raw.append(p.read_bytes())
    assert raw[0] == raw[1]


@pytest.mark.parametrize("d", DIMS)
def test_first_points_are_linked_as_by_sequential_insertion(tmp_path, d):
    """Batches hold one point each up to 47 points, and a beam wider than the index
    finds every reachable point: level 0 is then the sequential insertion's, link by
    link (neighbour heuristic and pruning, hrnn.h:619-659, 682-806)."""
    n, M = 47, 4
    X = data.mixture(n, d, 3, 1.0, 9, 9)
    h = H.HRNN(d, n, M, 64, 100, 8)
    h.add_points(X)
    p = str(tmp_path / "s.idx")
    h.saveIndex(p)
    adj = idx.read_idx(p).adj0()
    lanes, fused = H.detect_l2_order()
    D = np.zeros((n, n), np.float32)
    for i in range(n):
        D[i] = port.l2_batch(np.repeat(X[i:i + 1], n, 0), X, lanes, fused)

    def pick(base, cand, most):
        cand = sorted(cand, key=lambda c: (D[base, c], c))
        if len(cand) < most:
            return cand
        kept = []
        for c in cand:
            if len(kept) == most:
                break
            if all(not D[c, k] < D[base, c] for k in kept):
                kept.append(c)
        return kept

    links = {0: []}
    for i in range(1, n):
        seen, todo = {0}, [0]
        while todo:
            for k in links[todo.pop()]:
                if k not in seen:
                    seen.add(k)
                    todo.append(k)
        kept = pick(i, seen, M)
        links[i] = kept[::-1]
        for k in kept:
            if len(links[k]) < 2 * M:
                links[k] = links[k] + [i]
            else:
                links[k] = pick(k, links[k] + [i], 2 * M)[::-1]
    for i in range(n):
        assert list(adj[i, 1:1 + (adj[i, 0] & 0xFFFF)]) == links[i], i
