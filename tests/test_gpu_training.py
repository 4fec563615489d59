"""Accuracy of the closure network's training steps."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_paths import _mix64

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


def _adam64(p0, feat, y, epochs, batch, lr, seed):
    """The training steps in float64.  Returns the parameters, a bound on what float32 changes in each, and how far
    the weights stay from a midpoint of bfloat16 (in float32 units) and the units from zero: within either the
    forward pass could go the other way."""
    n, p = len(y), p0.astype(np.float64)
    m1, v1, bound = np.zeros_like(p), np.zeros_like(p), np.zeros_like(p)
    u, t, midpoint, unit = 2.0 ** -24, 0, np.inf, np.inf
    cuts = np.cumsum([1152, 32, 1024, 32, 32])
    with np.errstate(over="ignore"):
        for _ in range(epochs * -(-n // batch)):
            k = np.uint64(t) * np.uint64(0x100000001) + np.arange(batch, dtype=np.uint64)
            idx = (_mix64(np.uint64(seed) ^ _mix64(k)) % np.uint64(n)).astype(np.int64)
            W1, b1, W2, b2, w3, b3 = np.split(p, cuts)
            bits = np.concatenate([W1, W2, w3]).astype(np.float32).view(np.uint32) & 0xffff
            midpoint = min(midpoint, np.abs(bits.astype(np.int64) - 0x8000).min())
            W1, W2, w3 = (O.bf16_round(a.astype(np.float32)).astype(np.float64) for a in (W1, W2, w3))
            W1, W2 = W1.reshape(32, 36), W2.reshape(32, 32)
            x, lab = feat[idx].astype(np.float64), y[idx].astype(np.float64)
            u1 = x @ W1.T + b1
            h1 = np.maximum(u1, 0)
            u2 = h1 @ W2.T + b2
            h2 = np.maximum(u2, 0)
            unit = min(unit, np.abs(u1).min(), np.abs(u2).min())
            z = h2 @ w3 + b3
            a = np.clip(z, 0, 1)
            d = np.where(((z < 0) & (lab > 0)) | ((z > 1) & (lab < 1)), z - lab, a - lab)

            def gradient(gz, W2, w3, x):
                d2 = gz[:, None] * w3 * (h2 > 0)
                d1 = (d2 @ W2) * (h1 > 0)
                return np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ gz,
                                       [gz.sum()]])
            g = gradient(2 * d / batch, W2, w3, x)
            # the same sums of magnitudes, with the error's size of that of the terms of z
            size = gradient(2 * (h2 @ np.abs(w3) + np.abs(b3) + lab) / batch, np.abs(W2), np.abs(w3), np.abs(x))
            t += 1
            m1, v1 = 0.9 * m1 + 0.1 * g, 0.999 * v1 + 0.001 * g * g
            root = np.sqrt(v1 / (1 - 0.999 ** t)) + 1e-8
            p = p - lr * (m1 / (1 - 0.9 ** t)) / root
            bound += 64 * u * lr * size / root + 2 * u * np.abs(p) + 16 * u * lr
    return p, bound, midpoint, unit


@pytest.mark.parametrize("n,batch,epochs,seed,init", [
    (200, 97, 1, 9, 3),  # three steps of four tiles, the last of one sample
    (40, 33, 2, 4, 3),  # two epochs of two steps
    (20000, 9601, 1, 6, 10)])  # three steps of 301 tiles, 296 blocks
def test_trained_parameters_match_float64(n, batch, epochs, seed, init):
    """Every parameter after several Adam steps, within 64 roundings of the terms of its gradients (and of the
    parameter and the update themselves): for most parameters below a thousandth of one step's change."""
    from self_b200 import closure as CL
    r = np.random.default_rng(n)
    feat = r.uniform(0, 1, (n, 36)).astype(np.float32)
    y = np.clip(2.0 * feat[:, 5] - 0.5, 0, 1).astype(np.float32)
    m = CL.ClosureMLP(seed=init)
    ref, bound, midpoint, unit = _adam64(m.params, feat, y, epochs, batch, 1e-3, seed)
    assert midpoint >= 8 and unit >= 1e-6  # (of the inputs)
    assert np.median(bound) < 1e-3 * 1e-3
    m.train(torch.from_numpy(feat).cuda(), torch.from_numpy(y).cuda(), epochs=epochs, batch=batch, lr=1e-3, seed=seed)
    assert (np.abs(m.params - ref) <= bound).all()
