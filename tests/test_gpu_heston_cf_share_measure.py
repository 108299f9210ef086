"""The Heston characteristic-function pricer where phi(-i) = S exp((r - q) t)
leaves the range in which a share measure is formed: below 1e-14 the price is
NaN, and where the factor overflows the price is what the oracle's arithmetic
gives, whatever route a well-conditioned option takes.

Bar of the pricer's own tests: 1e-9 x max(1, |price|), NaN for NaN.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(spot=100.0, strike=97.0, t=100.0, r=0.02, q=0.01, v0=0.04, kappa=1.5, theta=0.05,
            sigma=0.05, rho=-0.6)
# log phi(-i): -33.4, -35.4, -32.3 | -32.22, -32.19, -20 | 505, 685 | 805 | -32.8
EDGES = [dict(q=0.4), dict(t=10.0, r=0.0, q=4.0), dict(r=0.0, q=0.369), dict(r=0.0, q=0.3683),
         dict(r=0.0, q=0.368), dict(r=0.0, q=0.246), dict(r=5.0, q=0.0), dict(r=6.8, q=0.0),
         dict(r=8.0, q=0.0), dict(spot=1e-6, strike=1e-6, t=2.0, r=0.0, q=9.5),
         # -13.3, -13.5 | 672.6, 674.6
         dict(r=0.0, q=0.179), dict(r=0.0, q=0.181), dict(r=6.68, q=0.0), dict(r=6.7, q=0.0)]


@pytest.mark.parametrize("copies", (1, 400))  # four warps an option, one
def test_share_measure_limits_against_oracle(qk, oracle, copies):
    cases = [{**BASE, **e, "option_type": ot, "integration_steps": 1024, "integration_limit": 20.0}
             for e in EDGES for ot in (0, 1)]
    cols = {k: np.tile(np.array([c[k] for c in cases]), copies) for k in cases[0]}
    got = qk.heston_price_cf_batch(**cols).reshape(copies, len(cases))
    assert np.array_equal(got, np.broadcast_to(got[0], got.shape), equal_nan=True)
    for c, g in zip(cases, got[0]):
        want = oracle.heston_cf(*c.values())
        assert (np.isnan(g) and np.isnan(want)) or abs(g - want) <= 1e-9 * max(1.0, abs(want)), (c, g, want)
