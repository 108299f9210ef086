"""The surrogate's host pricing call where its routes meet: options that the
entry checks decide do not depend on the network.
"""

import numpy as np
import pytest

from quantkernel_b200.surrogate import N_PARAMS, HestonSurrogate, sample_box

pytestmark = pytest.mark.gpu


def _quotes(n):
    """In the box, expired, outside the box (Monte Carlo) and refused, in turn."""
    b = sample_box(n, 23)
    ot = (np.arange(n) % 2).astype(np.int32)
    kind = np.arange(n) % 4 if n < 100 else np.where(np.arange(n) % 5000 < 8, np.arange(n) % 4, 0)
    b["t"][kind == 1] = 0.0
    b["strike"][kind == 2] *= 3.0
    b["v0"][kind == 3] = -0.01
    return b, ot, kind


@pytest.mark.parametrize("value", (np.nan, np.inf))
def test_decided_options_do_not_depend_on_the_network(qk, value):
    sur = HestonSurrogate(qk, seed=3)
    b, ot, kind = _quotes(64)
    want, src = sur.price_batch(**b, option_type=ot, fallback_paths=1000, fallback_steps=8)
    sur.set_parameters(np.full(N_PARAMS, value))
    got, src2 = sur.price_batch(**b, option_type=ot, fallback_paths=1000, fallback_steps=8)
    assert np.array_equal(src, src2)
    assert np.array_equal(src, np.array([0, 2, 1, 2])[kind])
    decided = kind != 0
    assert np.array_equal(got[decided], want[decided], equal_nan=True)
    assert np.all(np.isfinite(got[kind == 1])) and np.all(np.isfinite(got[kind == 2]))
    sur.close()
