"""The surrogate's row kernel at the edges of its tiling (64-row tiles, one CTA per SM over
several tiles, 65,536-row inference launches) and of the gradient's row splits (1024).

Tolerances as for the network's other tests (tests/test_surrogate_gpu.py): the oracle
rounds to bfloat16 where the kernels store it, so what is left is float32 accumulation
and the rare value that accumulation moves across a rounding boundary.
"""
import numpy as np
import pytest

from oracle import mlp
from cgppd_gb300 import surrogate as sg
from test_surrogate_gpu import pose_like, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 152 * 64 + 1, 65536 + 3])
def test_predictions_at_tile_edges(n):
    s = sg.Surrogate(batch=128, seed=9)
    X = pose_like(np.random.default_rng(n), n)
    out = s.predict(X)
    some = np.unique(np.concatenate([np.arange(min(n, 70)), np.arange(max(0, n - 70), n),
                                     np.random.default_rng(1).integers(0, n, 100)]))
    ref, _ = mlp.forward(s.params.astype(np.float64), X[some], bf16_path=True)
    assert np.max(np.abs(out[some] - ref)) <= 2e-3 * (1 + np.max(np.abs(ref)))
    s.close()


@pytest.mark.parametrize("n", [128, 384, 1024, 2048])
def test_gradients_at_split_edges(n):
    s = sg.Surrogate(batch=2048, seed=11)
    rng = np.random.default_rng(n)
    X, y = pose_like(rng, n), rng.normal(size=n).astype(np.float32)
    loss, g = s.loss_grad(X, y)
    alone, none = s.loss_grad(X, y, grad=False)
    assert none is None and alone == loss
    lb, gb = mlp.loss_grad(s.params.astype(np.float64), X, y, bf16_path=True)
    assert loss == pytest.approx(lb, rel=2e-3)
    for k, (o, m) in mlp.OFF.items():
        assert rel_err(g[o:o + m], gb[o:o + m]) < 2e-2, (k, rel_err(g[o:o + m], gb[o:o + m]))
    s.close()


def test_saturated_units():
    """Pre-activations of thousands on both sides (exp overflows and vanishes): the
    activations are z and -0, and nothing is lost on the way."""
    s = sg.Surrogate(batch=128, seed=13)
    p = s.params * np.float32(400.0)
    s.params = p
    X = pose_like(np.random.default_rng(5), 128)
    ref, _ = mlp.forward(p.astype(np.float64), X, bf16_path=True)
    out = s.predict(X)
    assert np.all(np.isfinite(out))
    assert np.max(np.abs(out - ref)) <= 2e-3 * (1 + np.max(np.abs(ref)))
    s.close()


def shuffled(n, seed):
    """The sequential shuffle of 0..n-1 with splitmix64, as the training order is defined."""
    mask, s = (1 << 64) - 1, (seed ^ 0x7A11) & ((1 << 64) - 1)
    p = list(range(n))
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        p[i], p[j] = p[j], p[i]
    return p


@pytest.mark.parametrize("n", [128, 129, 200, 1025, 5000, 152 * 1024 + 7])
def test_training_order_is_the_sequential_shuffle(n):
    """Targets that are all zero but for the row number: the mean squared error of a batch of
    a network that predicts zero names its rows.  (A learning rate that leaves the
    parameters where they are; history holds the mean over every 16th batch and the last.)"""
    s = sg.Surrogate(batch=128, seed=17)
    s.params = np.zeros(sg.N_PARAMS, np.float32)
    y = (1.0 + np.arange(n, dtype=np.float64) / n).astype(np.float32)
    s.add_samples(pose_like(np.random.default_rng(2), n), y)
    hist = s.train(1, lr=1e-30, clip=25.0, val_fraction=0.0)
    p, nb = shuffled(n, 17), n // 128
    logged = [b for b in range(nb) if b % 16 == 0 or b == nb - 1]
    want = np.sqrt(np.mean([np.mean(y[p[128 * b:128 * b + 128]].astype(np.float64) ** 2) for b in logged]))
    # 128-term float sums and the float32 mean: a few times 2^-24; another order of n rows
    # differs by about 1e-2 / sqrt(batches)
    assert hist[0, 0] == pytest.approx(want, rel=2e-6)
    s.close()
