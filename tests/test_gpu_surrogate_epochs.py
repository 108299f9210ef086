"""Every epoch of a training call sees each row of the dataset once, whatever
the next epoch's shuffle does meanwhile.

With a learning rate of zero and an untouched network the loss of a row is its
squared residual, so an epoch over all rows has the mean of those as its loss.
A row's residual is 1, 2, 4, ... 128 by its index mod 8 (mean square 2731, its
deviation 5800): m rows drawn again in place of others move the loss by about
sqrt(2 m) 5800 / (2731 n), which passes the bar from some hundred of the 2^18 rows on.
FP32 sums of 1024 terms (chains of four, a tree of eight levels, the division)
and the residuals' own rounding stay below 2^-19; steps are averaged in FP64.
"""

import numpy as np
import pytest

from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epochs", (1, 6))
def test_each_row_once_an_epoch(qk, epochs):
    n = 1 << 18
    f = features_of(**sample_box(n, 7))
    sur = HestonSurrogate(qk, seed=3)
    base = sur.predict(f)  # an untrained network is its base
    residual = 2.0 ** (np.arange(n) % 8)
    sur.set_dataset(f, base + residual)
    want = np.mean(residual.astype(np.float64) ** 2)
    for seed in (0, 1):
        losses = sur.train(epochs, batch=1024, lr=0.0, shuffle_seed=seed)
        assert np.all(np.abs(losses / want - 1.0) <= 2.0**-19), losses / want - 1.0
    sur.close()
