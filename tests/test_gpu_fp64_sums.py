"""Sums of the FP64 families where path factors could be far above the payoffs:
double-double sums of equal payoffs are exact, so a put whose paths all end
below the last bit of its strike (S_T = S exp(-g)) is worth its strike to that bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a full 53-bit significand, at either end of a power of two
STRIKES = (float.fromhex("0x1.fffffffffffffp+6"), float.fromhex("0x1.5555555555555p+6"),
           float.fromhex("0x1.0000000000001p+0"))


@pytest.mark.parametrize("model", ("standard_monte_carlo", "antithetic_variates", "importance_sampling",
                                   "quasi_monte_carlo_sobol", "quasi_monte_carlo_halton",
                                   "stratified_sampling"))
@pytest.mark.parametrize("paths", (1 << 14, 1 << 20))
def test_equal_payoffs_sum_exactly(qk, model, paths):
    grid = [(k, g) for k in STRIKES for g in (45.0, 60.0, 150.0, 290.0)]
    n = len(grid)
    cols = dict(spot=np.full(n, 100.0), strike=np.array([k for k, _ in grid]), t=np.ones(n),
                vol=np.full(n, 1e-3), r=np.zeros(n), q=np.array([g for _, g in grid]),
                option_type=np.ones(n, np.int32), paths=np.full(n, paths, np.int32))
    if model == "importance_sampling":
        cols["shift"] = np.zeros(n)
    if not model.startswith("quasi"):
        cols["seed"] = np.arange(n, dtype=np.uint64)
    price, _ = getattr(qk, model + "_price_se_batch")(**cols)
    assert np.array_equal(price, cols["strike"]), price - cols["strike"]
