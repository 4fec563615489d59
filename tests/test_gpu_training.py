"""Accuracy of the closure network's training steps."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_gradient_sums_of_a_large_batch_keep_float32_accuracy():
    """One Adam step on 2^22 copies of one sample.  With gradients far below Adam's epsilon the update is linear in
    them, so a parameter that starts at zero shows its gradient to a few roundings; a sum of 4 194 304 equal values
    over 131 072 tiles of 32, 443 to a block, passes through at most 7 + 443 + 12 + 3 roundings (one chain over a
    block's samples drifts by 1.4e-4 here)."""
    from self_b200 import closure as CL
    w3, y, f1 = 2.0 ** -40, np.float32(0.7), np.float32(0.9)
    W1, W2 = np.zeros((32, 36), np.float32), np.zeros((32, 32), np.float32)
    W1[:, 0] = W2[:, 0] = 1.0  # every unit's activation is 1
    z = np.zeros(32, np.float32)
    m = CL.ClosureMLP(params=np.concatenate([W1.ravel(), z, W2.ravel(), z, z + np.float32(w3), [0.0]]))
    x = np.zeros((1, 36), np.float32)
    x[0, :2] = 1.0, f1
    m.train(torch.from_numpy(x).cuda(), torch.full((1,), float(y), device="cuda"), epochs=1, batch=1 << 22, lr=1.0)
    g1, gb1, g2, gb2, _, _ = m.unpack()

    def gradient(p):
        u = -p.astype(np.float64)  # lr = 1: g / (|g| + eps)
        return u * float(np.float32(1e-8)) / (1.0 - np.abs(u))

    d2 = 2.0 * (32 * w3 - float(y)) * w3
    tol = 475 * 2.0 ** -24
    for got, ref in ((gb2, d2), (g2[:, 1], d2), (gb1[:1], 32 * d2), (g1[:1, 1], 32 * d2 * float(f1))):
        assert np.abs(gradient(got) / ref - 1.0).max() < tol
