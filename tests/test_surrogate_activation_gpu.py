"""The network's activation and its slope, unit by unit, against float64.

With every other weight zero the pre-activations of layer 4 are its biases, bit for bit:
the output weights' gradient then is 128 dO bf16(silu(z)) and, with unit output weights,
the biases' gradient 128 bf16(dO silu'(z)), both exact sums of 128 equal BF16 values.

Bounds: CUDA states 2 + floor(1.173 |x|) units for __expf(x), half a unit each for the
sum, the division and every product after it.  A BF16 result must be one that rounding
a value within that bound can give (for nearly every z exactly one).
"""
import numpy as np
import pytest

from oracle import mlp
from cgppd_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu

ROWS, TINY = 128, 1e-35  # past z = -88 exp(-z) overflows: silu and its slope become 0


def silu_inverse(h):
    """z >= 0 with silu(z) = h (bisection)."""
    lo, hi = np.zeros_like(h), h + 1.0
    for _ in range(80):
        m = 0.5 * (lo + hi)
        up = mlp.silu(m) < h
        lo, hi = np.where(up, m, lo), np.where(up, hi, m)
    return lo


def values(kind):
    rng = np.random.default_rng(3)
    if kind == "dense":
        return np.linspace(-12.0, 12.0, 256 * 8)
    if kind == "wide":
        return np.concatenate([rng.uniform(-87.0, 87.0, 256 * 3), rng.normal(scale=1e-3, size=128),
                               rng.uniform(-1e4, 1e4, 128)])
    if kind == "halves":  # silu within a few units of the middle between two BF16 values
        h = mlp.bf16(np.exp(rng.uniform(np.log(1e-3), np.log(60.0), 64))).astype(np.float32)
        z = silu_inverse((h.view(np.uint32) + np.uint32(0x8000)).view(np.float32).astype(np.float64)).astype(np.float32)
        return (z.view(np.uint32)[:, None] + np.arange(-8, 8).astype(np.uint32)).view(np.float32).ravel()
    edge = np.float32([-80.0, -87.33654, -88.02969, -88.72284])  # the guard; ends of exp's range
    near = (edge.view(np.uint32)[:, None] + np.arange(-4, 4).astype(np.uint32)).view(np.float32).ravel()
    rest = rng.uniform(-110.0, -79.0, 256 - near.size - 4)
    return np.concatenate([near, rest, [0.0, -0.0, 1e30, -1e30]])


def sigmoid_error(z):
    """s = 1 / (1 + exp(-z)) in float64 and the bound on its absolute error in FP32."""
    with np.errstate(over="ignore"):
        e = np.exp(-z)
    s = 1.0 / (1.0 + e)
    return s, s * ((2.0 + 1.173 * np.abs(z)) * 2.0 ** -23 * (1.0 - s) + 2.0 ** -23)


def between(got, mid, err):
    lo, hi = mlp.bf16(mid - err - TINY), mlp.bf16(mid + err + TINY)
    ok = (lo <= got) & (got <= hi)
    return ok.all(), np.flatnonzero(~ok)[:4]


@pytest.mark.parametrize("kind", ["dense", "wide", "halves", "edges"])
def test_activation_and_slope(kind):
    s = sg.Surrogate(batch=ROWS, seed=1)
    X = np.random.default_rng(0).normal(size=(ROWS, 8)).astype(np.float32)
    b4, w5 = slice(mlp.OFF["b4"][0], mlp.OFF["b4"][0] + 256), slice(mlp.OFF["w5"][0], mlp.OFF["w5"][0] + 256)
    zs = np.asarray(values(kind), np.float32)
    zs = np.resize(zs, -(-zs.size // 256) * 256)
    for part in zs.reshape(-1, 256):
        z = part.astype(np.float64)
        sig, ds = sigmoid_error(z)
        p = np.zeros(sg.N_PARAMS, np.float32)
        p[b4] = part
        s.params = p
        _, g = s.loss_grad(X, np.full(ROWS, -64.0, np.float32))  # dO = 2 * 64 / 128
        ok, at = between(g[w5].astype(np.float64) / ROWS, z * sig, np.abs(z) * (ds + sig * 2.0 ** -23))
        assert ok, (part[at], g[w5][at] / ROWS, (z * sig)[at])

        # (larger values would leave their sum no room for a residual of 64)
        part = np.where(np.abs(part) > 1e4, np.float32(0.5), part)
        z = part.astype(np.float64)
        sig, ds = sigmoid_error(z)
        p[b4], p[w5] = part, 1.0
        s.params = p
        out = s.predict(X)
        y = out - np.float32(64.0)
        d = np.float32(2.0) * (out - y) / np.float32(ROWS)
        assert np.all(d == d[0])
        _, g = s.loss_grad(X, y)
        slope = sig * (1.0 + z * (1.0 - sig))
        err = ds * (np.abs(1.0 + z * (1.0 - sig)) + sig * np.abs(z)) + 2.0 ** -22 * sig * (1.0 + np.abs(z) * (1.0 - sig))
        ok, at = between(g[b4].astype(np.float64) / ROWS, d[0] * slope, d[0] * (err + 2.0 ** -24 * np.abs(slope)))
        assert ok, (part[at], g[b4][at] / ROWS, slope[at])
    s.close()
