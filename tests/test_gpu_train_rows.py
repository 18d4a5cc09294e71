"""The training kernels (mlp.cu: train_rows_kernel, weight_grad_kernel,
update_kernel) at row counts around their tiles (32 rows per CTA, splits of 512
rows): loss and gradients against the float64 oracle, with the tolerances of
test_gpu_learned.py (BF16 activations and gradients, relative rounding 2^-9 per
value), and one AdamW step against its formula on those gradients."""
import numpy as np
import pytest

import gain_mlp as gm

pytestmark = pytest.mark.gpu


def batch(n, seed):
    rng = np.random.default_rng(seed)
    X = np.empty((n, 65), np.float32)
    X[:, :64] = rng.normal(1.0, 2.0, (n, 64))
    X[:, 64] = rng.uniform(5, 50, n) / 255.0
    return X, rng.uniform(0, 1, (n, 64)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 513, 1100])
def test_gradients_at_tile_edges(gpulib, gpuctx, n):
    import torch
    tr = gpulib.Trainer(batch=1100, seed=n)
    params = tr.params()
    X, T = batch(n, n)
    d = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    g, loss = tr.grad(*d)
    blob = gm.join([gm.bf16_round(p) if p.ndim == 2 else p for p in gm.split(params)])
    wl, wg = gm.loss_and_grad(blob, gm.bf16_round(X), T.astype(np.float64))
    assert abs(loss - wl) <= 1e-2 * wl
    for name, a, b in zip(("W1", "b1", "W2", "b2", "W3", "b3"), gm.split(g), gm.split(wg)):
        assert np.linalg.norm(a - b) < 3e-2 * np.linalg.norm(b), name
    # a step: the loss before the update, and AdamW's first step from these gradients
    lr, wd = 1e-3, 1e-2
    got = tr.step(*d, lr=lr, weight_decay=wd)
    assert got == loss
    m1, m2, steps = tr.state()
    assert steps == 1
    assert np.allclose(m1, 0.1 * g, rtol=1e-5, atol=1e-12) and np.allclose(m2, 0.001 * g * g, rtol=1e-4, atol=1e-20)
    decay = gm.join([np.full(p.shape, wd if p.ndim == 2 else 0.0) for p in gm.split(params)])
    want = params - lr * decay * params - lr * g / (np.abs(g) + 1e-8)
    assert np.allclose(tr.params(), want, rtol=0, atol=2e-6)
    # repeated from the same state, bit for bit
    tr.set_params(params)
    tr.set_state(np.zeros_like(m1), np.zeros_like(m2), 0)
    first = tr.params()
    assert np.array_equal(first, params) and tr.step(*d, lr=lr, weight_decay=wd) == loss
    a = tr.params()
    tr.set_params(params)
    tr.set_state(np.zeros_like(m1), np.zeros_like(m2), 0)
    tr.step(*d, lr=lr, weight_decay=wd)
    assert np.array_equal(a, tr.params())
