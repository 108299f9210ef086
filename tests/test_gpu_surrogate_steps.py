"""The fused training pass at batch sizes where its split can go wrong -- one
tile of 128 rows, tile counts below, at and above the slab sums' groups of
sixteen -- against the FP64 oracle, and two models trained alike against each
other, bit for bit.

The gradient bars are those of the 256-row check: cosine > 0.995 and 5% in
norm per layer (bf16 weights and activations), the loss to 2%.
"""

import numpy as np
import pytest

from oracle import mlp_oracle as mo
from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu


def _model(qk, seed=3):
    sur = HestonSurrogate(qk, seed=seed)
    p = sur.parameters()
    p[-257:-1] = np.random.default_rng(10).normal(scale=1 / 16, size=256)
    sur.set_parameters(p)
    return sur


@pytest.mark.parametrize("n", (128, 384, 2048, 2176, 4224, 19456))
def test_gradients_at_tile_counts(qk, n):
    sur = _model(qk)
    f = features_of(**sample_box(n, 7))
    t = np.random.default_rng(9).uniform(0.0, 0.3, n)
    loss, g = sur.gradients(f, t)
    x = mo.bf16_bits_to_float(sur.feature_rows(f))[:, :9]
    loss_ref, g_ref = mo.loss_and_grads(sur.parameters(), x, t - mo.bsm_mean_var_base(f))
    assert abs(loss - loss_ref) <= 0.02 * loss_ref
    k = 0
    for name, shape in mo.SHAPES:
        m = int(np.prod(shape))
        a, r = g[k:k + m], g_ref[k:k + m]
        k += m
        cos = float(a @ r / (np.linalg.norm(a) * np.linalg.norm(r)))
        rel = float(np.linalg.norm(a - r) / np.linalg.norm(r))
        assert cos > 0.995 and rel < 0.05, (name, cos, rel)


@pytest.mark.parametrize("rows,batch", ((640, 128), (5000, 384), (9000, 4224)))
def test_training_is_deterministic_over_calls(qk, rows, batch):
    """Two calls (the second starts at a step that need not be a multiple of
    its epoch) give the same losses and parameters on two models."""
    f = features_of(**sample_box(rows, 5))
    t = np.random.default_rng(4).uniform(0.0, 0.3, rows)
    out = []
    for _ in range(2):
        sur = _model(qk)
        sur.set_dataset(f, t)
        first = sur.train(2, batch=batch, shuffle_seed=1)
        second = sur.train(1, batch=batch, shuffle_seed=2)
        out.append((first, second, sur.parameters()))
        sur.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.all(np.isfinite(out[0][2])) and out[0][0][1] < out[0][0][0]
