"""Reverse-list segments of every size class of the sort (one to 32 registers per lane,
the block-wide sort beyond), narrow and wide entries, against the oracle's transpose."""
import numpy as np
import pytest

from oracle import port

import hrnn_b200 as H

pytestmark = pytest.mark.gpu

LENS = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2500]


def _graph(n, K, seed):
    """Every owner lists K distinct targets; target t < len(LENS) is listed LENS[t] times,
    at random ranks."""
    r = np.random.default_rng(seed)
    ids = np.stack([r.choice(np.arange(len(LENS), n), K, replace=False) for _ in range(n)]).astype(np.uint32)
    for t, m in enumerate(LENS):
        own = r.choice(n, m, replace=False)
        own = own[(ids[own] >= len(LENS)).any(1)]
        for o in own:
            free = np.nonzero(ids[o] >= len(LENS))[0]
            ids[o, r.choice(free)] = t
    cnt = r.integers(1, K + 1, n).astype(np.uint32)
    cnt[r.random(n) < 0.7] = K
    return ids, cnt


@pytest.mark.parametrize("K", [24, 1])
def test_noalloc_segments(K):
    import torch
    n = 4000
    ids, cnt = _graph(n, K, K) if K > 1 else (np.minimum(np.arange(n) // 1300, 2).astype(np.uint32)[:, None],
                                              np.ones(n, np.uint32))
    off, ent, rb, wide = port.rknng(ids, cnt, n, K)
    di, dc = torch.from_numpy(ids.view(np.int32)).cuda(), torch.from_numpy(cnt.view(np.int32)).cuda()
    do = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    de = torch.zeros(len(ent), dtype=torch.int32, device="cuda")
    got = H.build_rknng_noalloc(di.data_ptr(), dc.data_ptr(), n, K, do.data_ptr(), de.data_ptr(), len(ent))
    assert got == (rb, wide, len(ent))
    assert np.array_equal(do.cpu().numpy().view(np.uint64), off)
    assert np.array_equal(de.cpu().numpy().view(np.uint32), ent)


@pytest.mark.parametrize("wide", [False, True])
def test_index_segments(monkeypatch, wide):
    n, K = 4000, 24
    ids, cnt = _graph(n, K, 5)
    off, ent, rb, _ = port.rknng(ids, cnt, n, K)
    if wide:
        monkeypatch.setenv("HRNN_RKNNG_WIDE", "1")
    h = H.HRNN(16, n, 8, 20, 100, K)
    h.add_points(np.random.default_rng(0).standard_normal((n, 16)).astype(np.float32))
    h.refineKNNG(0, 1)
    h.set_knng(ids, np.zeros((n, K), np.float32), cnt)
    h.buildRKNNG()
    go, ge, grb, gw = h.get_rknng()
    assert (grb, gw) == (rb, wide)
    assert np.array_equal(go, off) and np.array_equal(ge.astype(np.uint64), ent.astype(np.uint64))
