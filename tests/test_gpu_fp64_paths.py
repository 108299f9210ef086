"""The FP64 Monte Carlo families at the sizes where their loops can go wrong --
ragged last quads of four paths, tiles one path short or long, several units
per thread -- and with constants on both sides of the range that the bounded
FP64 functions serve, against the oracle's FP64 replay of the same points.

Bars as for the same replay elsewhere: 2e-11 of the price's scale for the
terminal models, 1e-12 relative + 1e-12 of it for the variance-reduction ones
(1e-10 relative for quasi-Monte Carlo), standard errors to 1e-9.
"""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATHS = (3, 4, 5, 8, 511, 512, 513, 2049, 32767, 65537, 131077)

# in range; then a path factor above e^300, a spot below 1e-100, a strike above 1e20
CONSTANTS = (dict(spot=100.0, strike=103.0, vol=0.35, t=0.8),
             dict(spot=100.0, strike=103.0, vol=12.0, t=9.0),
             dict(spot=3e-101, strike=2.5e-101, vol=0.3, t=1.1),
             dict(spot=2e20, strike=1.9e20, vol=0.25, t=1.7))


@pytest.mark.parametrize("model", (0, 1, 5, 8, 9, 10, 11, 12))
def test_ragged_sizes_and_both_ranges(qk, oracle, model):
    cases = [dict(CONSTANTS[0], paths=p) for p in PATHS]
    cases += [dict(c, paths=p) for c in CONSTANTS[1:] for p in (5, 2049)]
    n = len(cases)
    col = lambda k, t=np.float64: np.array([c[k] for c in cases], t)  # noqa: E731
    seed = np.arange(n, dtype=np.uint64) * np.uint64(7919) + np.uint64(1 << 40)
    shift = np.where(np.arange(n) % 2 == 0, 0.4, -0.7)
    ot = (np.arange(n) % 2).astype(np.int32)
    plan = qk.plan(model=np.full(n, model, np.int32), spot=col("spot"), strike=col("strike"),
                   t=col("t"), vol=col("vol"), r=np.full(n, 0.03), q=np.full(n, 0.01), v0=shift,
                   option_type=ot, paths=col("paths", np.int32), seed=seed)
    plan.execute()
    price, se = plan.results()
    plan.close()
    for i, c in enumerate(cases):
        args = dict(c, r=0.03, q=0.01, option_type=int(ot[i]), seed=int(seed[i]))
        if model < 8:
            want, want_se = oracle.philox_price(model, steps=1, antithetic=model != 5, **args)
        else:
            want, want_se = oracle.philox_vr_price(model, shift=float(shift[i]), **args)
        scale = max(c["spot"], abs(want))
        if model < 8:
            tol = 2e-11 * scale
        elif model < 11:
            tol = 1e-12 * abs(want) + 1e-12 * scale
        else:
            tol = 1e-10 * scale
        assert abs(price[i] - want) <= tol, (model, c, price[i], want)
        if math.isfinite(want_se):
            assert abs(se[i] - want_se) <= 1e-9 * max(want_se, 1e-3 * scale), (model, c, se[i], want_se)
        else:
            assert not math.isfinite(se[i]), (model, c, se[i])
