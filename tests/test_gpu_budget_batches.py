"""Budget network at batch sizes around the kernels' tiles and row ranges: logits and
gradients against the FP64 oracle."""
import numpy as np
import pytest

from oracle import mlp

import hrnn_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [2, 15, 16, 17, 31, 33, 63, 65, 127, 129, 1023, 1025, 4097])
def test_logits_and_gradients(B):
    params = mlp.init_params(B)
    h = H.HRNN(32, 16, 8, 32, 100, 8)
    h.budget_set_weights(params)
    rng = np.random.default_rng(B)
    X = rng.standard_normal((B, 256)).astype(np.float32)
    Y = rng.integers(0, 2, (B, 2)).astype(np.uint8)
    # BF16 operands as on the device, FP64 sums here and FP32 there: 1e-6 a sum, and
    # an operand that rounds the other way moves a logit by at most 2e-3
    assert np.max(np.abs(h.budget_predict(X) - mlp.forward(params, X, bf16_ops=True)[4])) <= 2e-3
    ref_loss, ref = mlp.loss_and_grads(params, X, Y, bf16_ops=True)
    for _ in range(2):  # the second evaluation reuses the first one's buffers
        grads, loss = h.budget_gradients(X, Y)
        assert abs(loss - ref_loss) <= 1e-5 * max(1.0, abs(ref_loss))
        for t, (g, r) in enumerate(zip(grads, ref)):
            assert np.linalg.norm(g - r) <= 1e-3 * max(np.linalg.norm(r), 1e-30), t
