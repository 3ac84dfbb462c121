"""Budget network after a batch whose workspace did not fit the device: the next, smaller
batch gets one of its own."""
import numpy as np
import pytest

from oracle import mlp

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


def test_gradients_after_out_of_memory():
    import torch
    params = mlp.init_params(5)
    h = H.HRNN(32, 16, 8, 32, 100, 8)
    h.budget_set_weights(params)
    rng = np.random.default_rng(5)

    def check(B):
        X = rng.standard_normal((B, 256)).astype(np.float32)
        Y = rng.integers(0, 2, (B, 2)).astype(np.uint8)
        grads, _ = h.budget_gradients(X, Y)
        for t, (g, r) in enumerate(zip(grads, mlp.loss_and_grads(params, X, Y, bf16_ops=True)[1])):
            assert np.linalg.norm(g - r) <= 1e-3 * max(np.linalg.norm(r), 1e-30), (B, t)

    check(70)
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
    try:  # 268 MB of features fit, 1.9 GB of activations do not
        with pytest.raises(H.HrnnError) as e:
            h.budget_gradients(np.zeros((1 << 18, 256), np.float32), np.zeros((1 << 18, 2), np.uint8))
        assert e.value.code == H.ERR_NOMEM
        check(70)
    finally:
        del held
        torch.cuda.empty_cache()
    check(200)
