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
