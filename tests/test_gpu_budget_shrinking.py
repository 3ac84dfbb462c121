"""Budget network on one handle whose batches get smaller: gradients after a larger batch
made the workspace, against the FP64 oracle."""
import numpy as np
import pytest

from oracle import mlp

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,then", [(1025, [1024, 65, 2]), (1200, [1000]), (2049, [2048, 1281, 1280])])
@pytest.mark.parametrize("how", ["gradients", "predict"])
def test_gradients_after_a_larger_batch(first, then, how):
    params = mlp.init_params(first)
    h = H.HRNN(32, 16, 8, 32, 100, 8)
    h.budget_set_weights(params)
    rng = np.random.default_rng(first)
    for B in [first] + then:
        X = rng.standard_normal((B, 256)).astype(np.float32)
        Y = rng.integers(0, 2, (B, 2)).astype(np.uint8)
        if B == first and how == "predict":
            h.budget_predict(X)
            continue
        grads, loss = h.budget_gradients(X, Y)
        # as for fresh handles: BF16 operands, FP64 sums here and FP32 there
        ref_loss, ref = mlp.loss_and_grads(params, X, Y, bf16_ops=True)
        assert abs(loss - ref_loss) <= 1e-5 * max(1.0, abs(ref_loss)), B
        for t, (g, r) in enumerate(zip(grads, ref)):
            assert np.linalg.norm(g - r) <= 1e-3 * max(np.linalg.norm(r), 1e-30), (B, t)
