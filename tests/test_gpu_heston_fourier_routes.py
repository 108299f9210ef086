"""The Heston Fourier pricers' two routes -- bounded functions on
well-conditioned options, the general form on the rest -- and their two work
splits (four warps an option, one warp an option) at the sizes and parameters
where they meet, against the oracle.

Bars of the pricers' own tests: 1e-9 x max(1, |price|) for the
characteristic-function price, the same plus DBL_EPSILON times the oracle's
rounding scale for COS.  The split must not change a bit.
"""

import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(spot=100.0, strike=97.0, t=0.8, r=0.02, q=0.01, v0=0.04, kappa=1.5, theta=0.05,
            sigma=0.5, rho=-0.6)
# each at, just inside or just outside a limit of the bounded route
EDGES = [dict(), dict(sigma=0.02), dict(sigma=0.0199), dict(kappa=0.01, theta=0.04),
         dict(kappa=0.0099), dict(kappa=0.36, sigma=0.7, rho=0.5), dict(kappa=0.36, sigma=0.7, rho=0.49),
         dict(kappa=0.3, sigma=0.7, rho=0.5), dict(rho=0.9999), dict(rho=-0.99995), dict(t=100.0),
         dict(t=101.0), dict(t=1e-6), dict(t=9e-7), dict(v0=0.0, theta=0.0), dict(theta=10.0),
         dict(theta=10.5), dict(v0=10.5), dict(r=10.5, t=0.01), dict(spot=2e9, strike=2e9),
         dict(sigma=9.9, t=0.05), dict(sigma=5.0, t=1.2), dict(sigma=10.5, t=0.05)]
COUNTS = (16, 64, 65, 128, 191, 1024, 2100)


def _cols(cases):
    return {k: np.array([c[k] for c in cases]) for k in cases[0]}


@pytest.mark.parametrize("method", ("cf", "cos"))
def test_routes_against_oracle_and_splits_bit_for_bit(qk, oracle, method):
    last, size = ("integration_limit", 120.0) if method == "cf" else ("truncation_width", 10.0)
    count = "integration_steps" if method == "cf" else "n_terms"
    cases = [{**BASE, **e, "option_type": i % 2, count: 256 if method == "cos" else 1024, last: size}
             for i, e in enumerate(EDGES)]
    cases += [{**BASE, "option_type": i % 2, count: c, last: size} for i, c in enumerate(COUNTS)]
    cases += [{**BASE, "option_type": 0, count: 64, last: x} for x in (0.5, 1.0, 2000.0)]
    fn = qk.heston_price_cf_batch if method == "cf" else qk.cos_method_fang_oosterlee_heston_price_batch
    cols = _cols(cases)
    few = fn(**cols)
    reps = 3000 // len(cases) + 1  # enough options for one warp each
    many = fn(**{k: np.tile(v, reps) for k, v in cols.items()})
    assert np.array_equal(np.tile(few, reps), many, equal_nan=True)
    for c, got in zip(cases, few):
        args = [c[k] for k in ("spot", "strike", "t", "r", "q", "v0", "kappa", "theta", "sigma", "rho",
                               "option_type", count, last)]
        want = oracle.heston_cf(*args) if method == "cf" else oracle.heston_cos(*args)
        tol = 1e-9 * max(1.0, abs(want))
        if method == "cos":
            tol += sys.float_info.epsilon * oracle.heston_cos_error_scale(*args)
        assert (np.isnan(got) and np.isnan(want)) or abs(got - want) <= tol, (c, got, want)
