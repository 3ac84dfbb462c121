"""Caller-owned transpose where n K reaches 2^32 and the scatter's cursors take 8 bytes:
short rows in a table of that size, narrow and wide entries."""
import numpy as np
import pytest

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2048, 2100])
def test_transpose_of_a_table_of_4g_places(K):
    import torch
    n, deg = 1 << 21, 3
    g = torch.Generator(device="cuda").manual_seed(K)
    t = torch.randint(n, (n, deg), generator=g, device="cuda", dtype=torch.int32)
    t[:3000, 2] = 7  # a segment for the block-wide sort
    cnt = torch.randint(deg + 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    cnt[:3000] = deg
    ids = torch.empty(n * K, dtype=torch.int32, device="cuda")
    ids.view(n, K)[:, :deg] = t
    c, th = cnt.cpu().numpy(), t.cpu().numpy()
    own, rank = np.nonzero(np.arange(deg)[None, :] < c[:, None])
    target = th[own, rank]
    order = np.lexsort((own, rank, target))
    off = np.concatenate([[0], np.cumsum(np.bincount(target, minlength=n))])
    rb = int(K - 1).bit_length()
    want = (own[order].astype(np.uint64) << np.uint64(rb)) | rank[order].astype(np.uint64)
    do = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    de = torch.zeros(len(want), dtype=torch.int64 if K > 2048 else torch.int32, device="cuda")
    got = H.build_rknng_noalloc(ids.data_ptr(), cnt.data_ptr(), n, K, do.data_ptr(), de.data_ptr(), len(want))
    assert got == (rb, K > 2048, len(want))
    ent = de.cpu().numpy()
    assert np.array_equal(do.cpu().numpy(), off)
    assert np.array_equal(ent.view(np.uint64 if K > 2048 else np.uint32).astype(np.uint64), want)
    del ids, t, cnt, do, de
    torch.cuda.empty_cache()
